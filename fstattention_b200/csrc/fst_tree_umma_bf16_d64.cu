// Instantiates the tcgen05 tree kernel for bf16, head_dim 64.
#include "fst_tree_umma.cuh"

namespace fst {
cudaError_t launch_tree_umma_bf16_d64(const AttnArgs &a, cudaStream_t stream) { return launch_tree_umma_d<__nv_bfloat16, 64>(a, stream); }
}  // namespace fst
