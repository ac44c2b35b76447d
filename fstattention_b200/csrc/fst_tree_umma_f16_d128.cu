// Instantiates the tcgen05 tree kernel for f16, head_dim 128.
#include "fst_tree_umma.cuh"

namespace fst {
cudaError_t launch_tree_umma_f16_d128(const AttnArgs &a, cudaStream_t stream) { return launch_tree_umma_d<__half, 128>(a, stream); }
}  // namespace fst
