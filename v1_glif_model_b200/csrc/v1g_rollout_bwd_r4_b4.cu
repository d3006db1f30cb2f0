// Backward rollout kernel: 4 receptor channels, rows of at most 4 batch values.
#include "v1g_rollout_bwd.cuh"

int v1g_launch_bwd_r4_b4(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st) {
  return proj ? launch_bwd<4, 4, true, false>(h, a, grid, smem, st) : launch_bwd<4, 4, false, false>(h, a, grid, smem, st);
}
