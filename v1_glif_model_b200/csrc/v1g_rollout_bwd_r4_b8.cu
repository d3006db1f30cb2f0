// Backward rollout kernel: 4 receptor channels, rows of 5 to 8 batch values.
#include "v1g_rollout_bwd.cuh"

int v1g_launch_bwd_r4_b8(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st) {
  if (pack)
    return proj ? launch_bwd<4, 8, true, true>(h, a, grid, smem, st) : launch_bwd<4, 8, false, true>(h, a, grid, smem, st);
  return proj ? launch_bwd<4, 8, true, false>(h, a, grid, smem, st) : launch_bwd<4, 8, false, false>(h, a, grid, smem, st);
}
