// Backward rollout, host side: loss tables over the saved spikes, plan, launch of the reverse sweep
// (v1g_rollout_bwd.cuh) and the return of the weight gradients in the caller's synapse order.
#include "v1g_rollout_bwd.cuh"

namespace {

// ---- loss preparation over the saved spikes ------------------------------------------------

// rate_coef[n] = rate_cost*ls*2*(m_n - target_n)/(N*B*T); loss[1] = rate loss
__global__ void __launch_bounds__(256) rate_loss_kernel(const int* __restrict__ spike_count,
                                                        const float* __restrict__ target, int N,
                                                        float inv_bt, float cost, float* rate_coef,
                                                        float* loss) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  float l = 0.f;
  if (n < N) {
    const float m = (float)spike_count[n] * inv_bt;
    const float dlt = m - target[n];
    rate_coef[n] = cost * 2.f * dlt / (float)N * inv_bt;
    l = dlt * dlt;
  }
  __shared__ float ws[8];
  for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += ws[w];
    atomicAdd(loss + 1, cost * s / (float)N);
  }
}

// Fano-factor loss of the population spike count in bins of `bin` steps (one block).
// sgrad[b*nbins + k] = dL/d(count of bin k, row b); loss[3] = synchrony loss.
__global__ void __launch_bounds__(256) sync_loss_kernel(const int* __restrict__ popcount, int T, int B,
                                                        int bin, int nbins, float cost, float target,
                                                        float* __restrict__ sgrad, float* loss) {
  extern __shared__ float sh[];  // counts [B*nbins], then mean[B], var[B], fano[B]
  float* cnt = sh;
  float* mean = sh + B * nbins;
  float* var = mean + B;
  float* fano = var + B;
  for (int i = threadIdx.x; i < B * nbins; i += blockDim.x) {
    const int b = i / nbins, k = i - b * nbins;
    int s = 0;
    for (int q = 0; q < bin; ++q) s += popcount[(k * bin + q) * B + b];
    cnt[i] = (float)s;
  }
  __syncthreads();
  if (threadIdx.x < B) {
    const int b = threadIdx.x;
    float m = 0.f;
    for (int k = 0; k < nbins; ++k) m += cnt[b * nbins + k];
    m /= (float)nbins;
    float v = 0.f;
    for (int k = 0; k < nbins; ++k) {
      const float d = cnt[b * nbins + k] - m;
      v += d * d;
    }
    v /= (float)nbins;
    mean[b] = m;
    var[b] = v;
    fano[b] = v / fmaxf(m, 1e-7f);
  }
  __syncthreads();
  float fbar = 0.f;
  for (int b = 0; b < B; ++b) fbar += fano[b];
  fbar /= (float)B;
  const float dl_df = cost * 2.f * (fbar - target) / (float)B;
  for (int i = threadIdx.x; i < B * nbins; i += blockDim.x) {
    const int b = i / nbins;
    const float m = mean[b], v = var[b];
    const float dv = 2.f * (cnt[i] - m) / (float)nbins;
    float df;
    if (m > 1e-7f)
      df = dv / m - v / (m * m) / (float)nbins;
    else
      df = dv / 1e-7f;
    sgrad[i] = dl_df * df;
  }
  if (threadIdx.x == 0) atomicAdd(loss + 3, cost * (fbar - target) * (fbar - target));
}

__global__ void __launch_bounds__(256) permute_add_kernel(const float* __restrict__ src,
                                                          const int32_t* __restrict__ perm,
                                                          float* __restrict__ dst, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[perm ? perm[i] : i] += src[i];
}

__global__ void finish_loss_kernel(float* acc, float* out) {
  if (threadIdx.x == 0) {
    acc[0] = acc[1] + acc[2] + acc[3];
    if (out)
      for (int i = 0; i < 4; ++i) out[i] = acc[i];
  }
}

}  // namespace

// internal_order: d_w_* are buffers in the library's own synapse order (presynaptic CSR for the
// recurrent and LGN sources, gather-table order for the background) that the kernel accumulates
// into directly; otherwise they are in the caller's order and filled through a permutation.
static int rollout_bwd_impl(V1GHandle* h, const V1GLossSpec* loss, const float* g_z, const float* g_v,
                            float* d_w_rec, float* d_w_lgn, float* d_w_bkg, float* loss_out,
                            bool internal_order, void* stream) {
  if (!h) return V1G_EINVAL;
  if (!h->tape_valid)
    return v1g_fail(h, V1G_ESTATE, "v1g_rollout_bwd needs a preceding v1g_rollout_fwd with save_for_bwd");
  cudaStream_t st = (cudaStream_t)stream;
  const V1GConfig& c = h->cfg;
  const int N = c.n_neurons, R = c.n_receptors, D = c.max_delay, S = c.n_syn_types;
  // a pass reads the slots of the steps tn-1 .. tn+D while other blocks already publish tn-2 .. tn-4, and the LGN
  // gradient of the pass before reads up to tn+4
  const int K = std::max(D + 5, 9);
  const int B = h->tape_B, T = h->tape_T;
  if (R != 4 && R != 5)
    return v1g_fail(h, V1G_ERANGE, "backward rollout is built for 4 or 5 receptor channels, got %d", R);
  V1GLossSpec ls;
  if (loss) ls = *loss; else ls = V1GLossSpec{nullptr, nullptr, 0.f, 0.f, 0.f, 1.f, 50, 1.f};
  const bool rate_groups = ls.n_rate_groups > 0;
  if (ls.rate_cost != 0.f && !ls.rate_target && !rate_groups)
    return v1g_fail(h, V1G_EINVAL, "rate_cost without rate_target or rate populations");
  const bool proj = S <= 8;
  const int C = proj ? S : R;
  const int BP = B <= 4 ? 4 : 8;
  const bool pack = (B == 5) && !h->opt_no_q_pack;  // five 24-bit floats per 16-byte row
  const int QW = pack ? 4 : BP;
  const int Np = (N + 31) & ~31;
  int rc;

  V1GRolloutPlan plan;
  v1g_plan_rollout(h, B, 1 + 2 * R, 0, 0, &plan);
  plan.chunkP = (plan.chunk + 3) & ~3;  // planes only need 16-byte alignment here
  if (plan.chunkP > 65535) return v1g_fail(h, V1G_ERANGE, "slice of %d neurons per block exceeds 65535", plan.chunkP);
  auto al = [](size_t b) { return (b + 15) & ~(size_t)15; };
  const size_t plane = (size_t)B * plan.chunkP;
  const bool meta = !h->opt_no_meta && h->src[V1G_SRC_REC].syn8 != nullptr && h->src[V1G_SRC_REC].nnz > 0;
  if (meta && (rc = v1g_build_bwd_records(h, st))) return rc;
  size_t smem = al(sizeof(float) * S * R) + al(sizeof(float) * PS * plane) + al(sizeof(float) * PS * B * c.n_bkg) +
                al(sizeof(int) * 8) +
                al(sizeof(unsigned long long) * 4) + al(sizeof(int4) * plan.chunkP) + al(sizeof(int) * (plan.chunkP + 1));
  // The L1 cache is what is left of the SM's 256 KB after the shared-memory carve-out, and it holds
  // the sectors of the gather's loads in flight: with less than ~60 KB of it the gather runs at half
  // speed.  What can also live in global memory therefore goes on chip only below 195 KB.
  const size_t on_chip = std::min<size_t>((size_t)h->smem_optin, 195 * 1024);
  const size_t tape_bytes = al(sizeof(float) * PS * plane);
  int tape_in_smem = 0;
  if (smem + tape_bytes <= on_chip) {
    tape_in_smem = 1;
    smem += tape_bytes;
  }
  const size_t state_bytes = al(sizeof(float) * plane * (1 + 2 * R));
  int state_in_smem = 0;
  if (!h->opt_force_global && smem + state_bytes <= on_chip) {
    state_in_smem = 1;
    smem += state_bytes;
  }
  int bkg_cap = 0;
  {
    const V1GSource& bk0 = h->src[V1G_SRC_BKG];
    for (int g = 0; g < plan.grid; ++g) {
      const int a0 = g * plan.chunk, a1 = std::min(N, a0 + plan.chunk);
      bkg_cap = std::max(bkg_cap, bk0.in_ptr_host[a1] - bk0.in_ptr_host[a0]);
    }
  }
  const size_t bkg_bytes = al(sizeof(int) * bkg_cap) + al(sizeof(float) * bkg_cap) + al(bkg_cap);
  int bkg_in_smem = 0;
  if (smem + bkg_bytes <= on_chip) {
    bkg_in_smem = 1;
    smem += bkg_bytes;
  }
  if (smem > (size_t)h->smem_optin)
    return v1g_fail(h, V1G_ERANGE, "backward rollout needs %zu B of shared memory per block", smem);
  if (!state_in_smem)
    if ((rc = v1g_reserve(h, &h->state_ws, &h->state_ws_cap, (int64_t)(plane * (1 + 2 * R) * plan.grid)))) return rc;

  // scratch: Q ring, CSR-order weight gradients, loss tables
  const int64_t q_elems = (int64_t)K * Np * C * QW;
  if (q_elems >= 0x7fffffffLL) return v1g_fail(h, V1G_ERANGE, "backward Q ring of %lld elements exceeds 32-bit indexing", (long long)q_elems);
  if ((rc = v1g_reserve(h, &h->dy_ring, &h->dy_ring_cap, q_elems))) return rc;
  const bool sync_samples = ls.sync_cost != 0.f && ls.n_sync_samples > 0;
  const int nbins = (ls.sync_cost != 0.f && !sync_samples && ls.sync_bin > 0) ? T / ls.sync_bin : 0;
  // loss scratch layout (floats): acc[4] | rate_coef[N] | sgrad[B*nbins] | spike_count[N] (int) | popcount[T*B] (int)
  const int64_t ls_elems = 4 + (int64_t)N + (int64_t)B * std::max(nbins, 1) + N + (int64_t)T * B;
  if ((rc = v1g_reserve(h, &h->loss_scratch, &h->loss_scratch_cap, ls_elems))) return rc;
  float* acc = h->loss_scratch;
  float* rate_coef = acc + 4;
  float* sgrad = rate_coef + N;
  int* spike_count = (int*)(sgrad + (int64_t)B * std::max(nbins, 1));
  int* popcount = spike_count + N;
  float* dw_int[V1G_NSRC] = {d_w_rec, d_w_lgn, d_w_bkg};
  for (int s = 0; s < V1G_NSRC; ++s) {
    if (internal_order && dw_int[s]) continue;  // the caller's buffer is accumulated into directly
    const int64_t nnz = std::max<int64_t>(h->src[s].nnz, 1);
    if (!h->dw_csr[s]) V1G_CUDA(h, cudaMalloc((void**)&h->dw_csr[s], (size_t)nnz * sizeof(float)));
    V1G_CUDA(h, cudaMemsetAsync(h->dw_csr[s], 0, (size_t)nnz * sizeof(float), st));
    dw_int[s] = h->dw_csr[s];
  }
  V1G_CUDA(h, cudaMemsetAsync(h->loss_scratch, 0, (size_t)ls_elems * sizeof(float), st));
  V1G_CUDA(h, cudaMemsetAsync(h->dy_ring, 0, (size_t)q_elems * sizeof(float), st));
  V1G_CUDA(h, cudaMemsetAsync(h->barrier, 0, V1G_BARRIER_BYTES, st));

  const bool want_rate = ls.rate_cost != 0.f, want_sync = nbins >= 1;
  if (want_rate || want_sync) {
    // spike counts per neuron and per (step, batch row) come from the forward kernel
    spike_count = h->tape_stats;
    popcount = h->tape_stats + N;
    v1g_count_launches(((want_rate && !rate_groups) ? 1 : 0) + (want_sync ? 1 : 0));
    if (want_rate && rate_groups) {
      if ((rc = v1g_rate_distribution_loss(h, &ls, spike_count, B, T, rate_coef, acc + 1, st))) return rc;
    } else if (want_rate) {
      rate_loss_kernel<<<(N + 255) / 256, 256, 0, st>>>(spike_count, ls.rate_target, N,
                                                       1.f / ((float)B * (float)T),
                                                       ls.rate_cost * ls.loss_scale, rate_coef, acc);
    }
    if (want_sync)
      sync_loss_kernel<<<1, 256, sizeof(float) * (B * nbins + 3 * B), st>>>(
          popcount, T, B, ls.sync_bin, nbins, ls.sync_cost * ls.loss_scale, ls.fano_target, sgrad, acc);
    V1G_CUDA(h, cudaGetLastError());
  }

  V1GSyncTables sync_tables;
  sync_tables.first = nullptr;
  if (sync_samples)
    if ((rc = v1g_sync_samples_loss(h, &ls, B, T, acc + 3, &sync_tables, st))) return rc;

  const float* osi_coef = nullptr;
  int osi_t0 = 0, osi_t1 = 0;
  if ((rc = v1g_osi_dsi_loss(h, &ls, B, T, acc + 3, &osi_coef, &osi_t0, &osi_t1, st))) return rc;

  BwdArgs a;
  a.sync = sync_tables;
  a.osi_coef = osi_coef; a.osi_t0 = osi_t0; a.osi_t1 = osi_t1;
  a.N = N; a.D = D; a.K = K; a.B = B; a.T = T;
  a.chunk = plan.chunk; a.chunkP = plan.chunkP; a.S = S; a.C = C; a.n_bkg = c.n_bkg;
  a.state_in_smem = state_in_smem;
  a.tape_in_smem = tape_in_smem;
  a.bkg_in_smem = bkg_in_smem;
  a.bkg_cap = bkg_cap;
  const V1GSource& rs = h->src[V1G_SRC_REC];
  const V1GSource& lsrc = h->src[V1G_SRC_LGN];
  const V1GSource& bk = h->src[V1G_SRC_BKG];
  a.rec_rowptr = rs.rowptr; a.rec_post = rs.post; a.rec_w = rs.w; a.rec_sid = rs.sid;
  a.rec_pad = meta ? rs.brec : nullptr;
  a.rec_brow = meta ? rs.brow : nullptr;
  a.rec_nnz = (int)rs.nnz;
  a.lgn_post = lsrc.post; a.lgn_sid = lsrc.sid;
  a.bkg_inptr = bk.in_ptr; a.bkg_inpre = bk.in_pre; a.bkg_insid = bk.in_sid;
  a.decay = h->decay; a.cf = h->cf; a.basis = h->basis;
  for (int r = 0; r < V1G_MAX_RECEPTORS; ++r) {
    a.sd[r] = r < R ? h->syn_decay[r] : 0.f;
    a.pinit[r] = r < R ? h->psc_initial[r] : 0.f;
    a.dtsd[r] = c.dt * a.sd[r];
  }
  a.lr_scale = c.lr_scale; a.vd_keep = h->vd_keep; a.rec_factor = h->rec_grad_factor;
  a.damp = c.dampening_factor; a.inv_width = 1.f / c.pseudo_width; a.gauss_std = c.gauss_std;
  a.gauss = (c.flags & V1G_FLAG_PSEUDO_GAUSS) ? 1 : 0;
  a.hard_reset = (c.flags & V1G_FLAG_HARD_RESET) ? 1 : 0;
  a.tape_v = h->tape_v;
  a.hist0 = h->tape_has_hist0 ? h->tape_hist0 : nullptr;
  a.lgn_off = h->lgn_offsets; a.lgn_ent4 = h->lgn_ent4; a.lgn_nseg = h->lgn_nseg;
  a.bkg_counts = h->tape_counts;
  a.rate_coef = want_rate ? rate_coef : nullptr;
  a.rate_t0 = rate_groups ? std::max(ls.rate_pre_delay, 0) : 0;
  a.rate_t1 = rate_groups ? T - std::max(ls.rate_post_delay, 0) : T;
  a.sgrad = want_sync ? sgrad : nullptr;
  a.sync_bin = ls.sync_bin; a.nbins = nbins;
  a.volt_coef = ls.voltage_cost * ls.loss_scale / ((float)B * (float)T * (float)N);
  a.volt_threshold_mode = ls.voltage_mode == 1 ? 1 : 0;
  a.v_lo = ls.v_lo;
  a.g_z = g_z; a.g_v = g_v;
  a.dw_rec = dw_int[V1G_SRC_REC]; a.dw_lgn = dw_int[V1G_SRC_LGN]; a.dw_bkg = dw_int[V1G_SRC_BKG];
  a.loss_acc = acc;
  a.Q = h->dy_ring; a.state_ws = h->state_ws;
  a.barrier = h->barrier; a.status = h->dev_status; a.counters = h->counters;
  a.spin_limit = h->opt_spin_limit;
  a.phase_ns = nullptr;
  if (h->opt_phase_timers) {
    if ((rc = v1g_reserve(h, &h->phase_ns, &h->phase_ns_cap, (int64_t)4 * plan.grid))) return rc;
    V1G_CUDA(h, cudaMemsetAsync(h->phase_ns, 0, sizeof(unsigned long long) * 4 * plan.grid, st));
    a.phase_ns = h->phase_ns;
    h->phase_grid = plan.grid;
  }
  // keep the Q ring resident in L2 (it is gathered at random, one sector per synapse and step)
  if (h->opt_l2_window) {
    cudaDeviceProp prop;
    V1G_CUDA(h, cudaGetDeviceProperties(&prop, h->device));
    const size_t q_bytes = (size_t)q_elems * sizeof(float);
    if (prop.persistingL2CacheMaxSize > 0 && prop.accessPolicyMaxWindowSize > 0) {
      const size_t carve = std::min<size_t>((size_t)prop.persistingL2CacheMaxSize, q_bytes);
      V1G_CUDA(h, cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, carve));
      cudaStreamAttrValue attr;
      attr.accessPolicyWindow.base_ptr = h->dy_ring;
      attr.accessPolicyWindow.num_bytes = std::min<size_t>(q_bytes, (size_t)prop.accessPolicyMaxWindowSize);
      attr.accessPolicyWindow.hitRatio = (float)std::min(1.0, (double)carve / (double)attr.accessPolicyWindow.num_bytes);
      attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
      attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
      V1G_CUDA(h, cudaStreamSetAttribute(st, cudaStreamAttributeAccessPolicyWindow, &attr));
    }
  }
  rc = (R == 4) ? (BP == 4 ? v1g_launch_bwd_r4_b4 : v1g_launch_bwd_r4_b8)(h, a, proj, pack, plan.grid, smem, st)
                : (BP == 4 ? v1g_launch_bwd_r5_b4 : v1g_launch_bwd_r5_b8)(h, a, proj, pack, plan.grid, smem, st);
  if (h->opt_l2_window) {
    cudaStreamAttrValue attr;
    attr.accessPolicyWindow.base_ptr = nullptr;
    attr.accessPolicyWindow.num_bytes = 0;
    attr.accessPolicyWindow.hitRatio = 0.f;
    attr.accessPolicyWindow.hitProp = cudaAccessPropertyNormal;
    attr.accessPolicyWindow.missProp = cudaAccessPropertyNormal;
    cudaStreamSetAttribute(st, cudaStreamAttributeAccessPolicyWindow, &attr);
  }
  if (rc) return rc;

  // weight gradients back to the caller's synapse order, accumulated
  const int blocks = h->n_sms * 8;
  if (internal_order) {
    finish_loss_kernel<<<1, 32, 0, st>>>(acc, loss_out);
    v1g_count_launches(1);
    V1G_CUDA(h, cudaGetLastError());
    return V1G_OK;
  }
  if (d_w_rec && rs.nnz) permute_add_kernel<<<blocks, 256, 0, st>>>(h->dw_csr[V1G_SRC_REC], rs.perm, d_w_rec, rs.nnz);
  if (d_w_lgn && lsrc.nnz) permute_add_kernel<<<blocks, 256, 0, st>>>(h->dw_csr[V1G_SRC_LGN], lsrc.perm, d_w_lgn, lsrc.nnz);
  if (d_w_bkg && bk.nnz) permute_add_kernel<<<blocks, 256, 0, st>>>(h->dw_csr[V1G_SRC_BKG], bk.in_perm, d_w_bkg, bk.nnz);
  finish_loss_kernel<<<1, 32, 0, st>>>(acc, loss_out);
  v1g_count_launches(1 + ((d_w_rec && rs.nnz) ? 1 : 0) + ((d_w_lgn && lsrc.nnz) ? 1 : 0) + ((d_w_bkg && bk.nnz) ? 1 : 0));
  V1G_CUDA(h, cudaGetLastError());
  return V1G_OK;
}

extern "C" int v1g_rollout_bwd(V1GHandle* h, const V1GLossSpec* loss, const float* g_z,
                               const float* g_v, float* d_w_rec, float* d_w_lgn, float* d_w_bkg,
                               float* loss_out, void* stream) {
  return rollout_bwd_impl(h, loss, g_z, g_v, d_w_rec, d_w_lgn, d_w_bkg, loss_out, false, stream);
}

extern "C" int v1g_rollout_bwd_internal(V1GHandle* h, const V1GLossSpec* loss, const float* g_z,
                                        const float* g_v, float* grads_flat, float* loss_out,
                                        void* stream) {
  if (!h) return V1G_EINVAL;
  if (!grads_flat) return v1g_fail(h, V1G_EINVAL, "v1g_rollout_bwd_internal: null gradient buffer");
  float* g0 = grads_flat;
  float* g1 = g0 + h->src[V1G_SRC_REC].nnz;
  float* g2 = g1 + h->src[V1G_SRC_LGN].nnz;
  return rollout_bwd_impl(h, loss, g_z, g_v, g0, g1, g2, loss_out, true, stream);
}
