// Instantiates the tcgen05 tree kernel for bf16, head_dim 128.
#include "fst_tree_umma.cuh"

namespace fst {
cudaError_t launch_tree_umma_bf16_d128(const AttnArgs &a, cudaStream_t stream) { return launch_tree_umma_d<__nv_bfloat16, 128>(a, stream); }
}  // namespace fst
