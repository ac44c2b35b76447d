// Instantiates the tcgen05 tree kernel for f16, head_dim 64.
#include "fst_tree_umma.cuh"

namespace fst {
cudaError_t launch_tree_umma_f16_d64(const AttnArgs &a, cudaStream_t stream) { return launch_tree_umma_d<__half, 64>(a, stream); }
}  // namespace fst
