// Fused backward rollout (BPTT): the reverse sweep over the T steps saved by v1g_rollout_fwd, in
// ONE persistent cooperative kernel with the same neuron slicing as the forward kernels.
//
// Adjoint recursion (g_* = dL/d(state after step t); reference: the custom gradients at
// models.py:58-64, 174-261 and the stop-gradients / straight-through factors at :994, 1010-1018,
// 1081), processed for t = T-1 .. 0:
//   g_z   = dl/dz(t) + rec_factor * sum over the out-synapses j of neuron n (delay d_j) of
//           w_j * sum_r basis[sid_j, r] * dy(t + d_j)[b, post_j, r]
//   g_v'  = dl/dv(t) + g_v + [r(t) == 0] * g_z * pseudo(v(t) - 1)        (hard reset: 0 if r(t) > 0)
//   g_v  <- decay * (1 - d_v) * g_v'              g_asc_k <- asc_decay_k * g_asc_k + cf * g_v'
//   g_p  <- sd * g_p + cf * g_v'                  g_pr   <- sd * g_pr + dt * sd * g_p(old)
//   dy(t)[b, n, r] = lr_scale * psc_initial_r * g_pr(t)
//   dW_rec[j] += sum_b z(t)[b, n] * sum_r basis[sid_j, r] * dy(t + d_j)[b, post_j, r]   (no dampening)
//   dW_lgn[j] += sum_b x(t)[b, pre_j] * (same with dy(t))      dW_bkg[j] += sum_b count(t)[b, pre_j] * (...)
//
// dy(t) only depends on g_pr(t+1) and g_p(t+1), which are final once step t+2 has been processed, and the
// gather of step t reads dy(t+1 .. t+D).  So with all steps > tn processed, dy(>= tn-1) is known, and the
// gathers of the THREE steps tn, tn-1, tn-2 can run before any of them is processed: a pass of the loop
//   loads the tape of the three steps and queues the rows that need a gradient,
//   waits until every block has finished the previous pass,
//   walks the queued rows once for all three steps (one warp per row),
//   processes the dense adjoint of the three steps, publishing dy(tn-2 .. tn-4).
// One step per pass costs three times the record reads, row overheads and barriers, and three separate
// requests where the ring rows of consecutive steps can share one.
//
// What is published is Q, a ring over K = max(D+5, 9) steps with a 16- or 32-byte row per (neuron, channel,
// step), the K steps of a channel next to each other:
//   projected mode (S <= 8 synapse types): Q[n][s][slot][b] = sum_r basis[s, r] * dy[b, n, r]; a synapse
//       then needs ONE row per step, Q[post][sid][slot of t+d][0..B)
//   raw mode: Q[n][slot][r][b] = dy[b, n, r]; the consumer contracts with basis[sid, :] (R rows)
// The three steps of a synapse read three consecutive rows (48 bytes): three lanes share a synapse, one per
// step, ten synapses per load instruction, so that a request fetches one or two lines for three steps.
//
// Measured (B200, 66,634 neurons, batch 5, 500 steps, us per reverse step), one step per pass with one lane
// per synapse -> three steps per pass: gather 33.3 -> 21.1, dense part 6.4 -> 6.0, whole kernel 43.4 -> 31.0.
// The old gather was bound by the L1's one line per cycle (54 k line accesses per step and SM); now L1 line
// accesses are down by a third, L2 sectors by a third and record reads by two thirds.
#pragma once

#include <algorithm>
#include <type_traits>

#include "v1g_rollout_common.cuh"

struct BwdArgs {
  int N, D, K, B, T, chunk, chunkP, S, C, n_bkg, state_in_smem, tape_in_smem, bkg_in_smem, bkg_cap;
  const int32_t *rec_rowptr, *rec_post;
  const float* rec_w;
  const uint8_t* rec_sid;
  int rec_nnz;
  // padded records of the gather {row of the ring | (delay-1) << 29, weight bits} and row starts in groups of
  // V1G_ROW_PAD (V1GSource::brec), or NULL
  const uint2* rec_pad;
  const int32_t* rec_brow;
  const int32_t* lgn_post;
  const uint8_t* lgn_sid;
  const int32_t *bkg_inptr, *bkg_inpre;
  const uint8_t* bkg_insid;
  const float *decay, *cf, *basis;
  float sd[V1G_MAX_RECEPTORS], pinit[V1G_MAX_RECEPTORS], dtsd[V1G_MAX_RECEPTORS];
  float lr_scale, vd_keep, rec_factor, damp, inv_width, gauss_std;
  int gauss, hard_reset;
  // saved forward
  const float* tape_v;
  const uint8_t* hist0;  // initial spike-history bits [B][N], or NULL for a zero initial state
  const int32_t* lgn_off;
  const uint4* lgn_ent4;  // {batch row << 24 | unit, first synapse, end, 0} per event
  int lgn_nseg;
  const int32_t* bkg_counts;
  // loss
  const float* rate_coef;  // [N] dL/dz contribution of the rate term, or NULL
  int rate_t0, rate_t1;    // steps whose spikes enter the rate term
  V1GSyncTables sync;      // synchrony target over given samples (first == NULL: off)
  const float* osi_coef;   // [B][N] dL/dz of the OSI/DSI target inside [osi_t0, osi_t1), or NULL
  int osi_t0, osi_t1;
  const float* sgrad;      // [B][nbins] dL/d(bin count), or NULL
  int sync_bin, nbins;
  float volt_coef;  // voltage_cost * loss_scale / (B*T*N); gradient is 2*volt_coef*(...)
  int volt_threshold_mode;
  const float* v_lo;
  const float *g_z, *g_v;  // explicit [B,T,N] gradients, nullable
  // outputs (accumulated)
  float *dw_rec, *dw_lgn, *dw_bkg;  // CSR order, CSR order, gather-table order
  float* loss_acc;                  // [4]; [2] += voltage loss
  // plumbing
  float* Q;
  float* state_ws;
  unsigned long long* barrier;
  int32_t* status;
  unsigned long long* counters;
  long long spin_limit;
  unsigned long long* phase_ns;
};

namespace {

#ifndef V1G_BWD_NT
#define V1G_BWD_NT 512
#endif
#ifndef V1G_BWD_GROUPS
#define V1G_BWD_GROUPS 5   // 10-synapse groups of a gather pass with one 16-byte row per lane
#endif
#ifndef V1G_BWD_GROUPS2
#define V1G_BWD_GROUPS2 4  // groups of a gather pass with 32 bytes per lane
#endif
#ifndef V1G_BWD_STAGES
#define V1G_BWD_STAGES 2   // Q-row buffers of the gather pipeline
#endif
constexpr int NT = V1G_BWD_NT;
constexpr int NW = NT / 32;
constexpr int BAR_TID = NT - 32;  // the thread that talks to the grid-wide phase counters

__device__ __forceinline__ unsigned long long gtime_b() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ float pseudo_h(float vs, const BwdArgs& a) {
  if (a.gauss) return expf(-(vs * vs) / (a.gauss_std * a.gauss_std)) * a.damp;
  float x = fabsf(vs);
  x = x * a.inv_width;
  return a.damp * fmaxf(1.f - x, 0.f);
}

// A Q row holds the values of all batch rows for one (neuron, channel): BP_ fp32 words, or - for a
// batch of exactly 5 - five 24-bit floats (sign, 8 exponent, 15 mantissa bits, round to nearest
// even: 7.6e-6 relative) packed into four words, which keeps the row at 16 bytes and the whole
// ring at half the size, inside L2.
__device__ __forceinline__ unsigned f24(float x) {
  unsigned u = __float_as_uint(x);
  u += 0x7fu + ((u >> 8) & 1u);
  return u >> 8;
}

__device__ __forceinline__ float4 pack_row5(const float (&v)[8]) {
  const unsigned r0 = f24(v[0]), r1 = f24(v[1]), r2 = f24(v[2]), r3 = f24(v[3]), r4 = f24(v[4]);
  uint4 w;
  w.x = r0 | (r1 << 24);
  w.y = (r1 >> 8) | (r2 << 16);
  w.z = (r2 >> 16) | (r3 << 8);
  w.w = r4;
  return make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
}

// the 16-byte words of a Q row -> its BP_ batch values
template <int BP_, bool PACK>
__device__ __forceinline__ void unpack_row(const float4 (&raw)[PACK ? 1 : BP_ / 4], float (&q)[BP_]) {
  const float4 a = raw[0];
  if (PACK) {
    const unsigned w0 = __float_as_uint(a.x), w1 = __float_as_uint(a.y), w2 = __float_as_uint(a.z),
                   w3 = __float_as_uint(a.w);
    q[0] = __uint_as_float(w0 << 8);
    q[1] = __uint_as_float(__funnelshift_l(w0, w1, 16) & 0xffffff00u);
    q[2] = __uint_as_float(__funnelshift_l(w1, w2, 24) & 0xffffff00u);
    q[3] = __uint_as_float(w2 & 0xffffff00u);
    q[4 % BP_] = __uint_as_float(w3 << 8);
#pragma unroll
    for (int b = 5; b < BP_; ++b) q[b] = 0.f;
    return;
  }
  q[0] = a.x; q[1] = a.y; q[2] = a.z; q[3] = a.w;
  if (BP_ == 8) {
    const float4 b = raw[(BP_ / 4 - 1) % (PACK ? 1 : BP_ / 4)];
    q[4 % BP_] = b.x; q[5 % BP_] = b.y; q[6 % BP_] = b.z; q[7 % BP_] = b.w;
  }
}

template <int BP_, bool PACK>
__device__ __forceinline__ void load_row(const float* p, float (&q)[BP_]) {
  float4 raw[PACK ? 1 : BP_ / 4];
#pragma unroll
  for (int v = 0; v < (PACK ? 1 : BP_ / 4); ++v) raw[v] = __ldcg((const float4*)p + v);
  unpack_row<BP_, PACK>(raw, q);
}

// one 32-byte pair row {Q(tau), Q(tau-1)} with a single load instruction
__device__ __forceinline__ void load_pair(const float* p, float4& lo, float4& hi) {
  asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(lo.x), "=f"(lo.y), "=f"(lo.z), "=f"(lo.w), "=f"(hi.x), "=f"(hi.y), "=f"(hi.z), "=f"(hi.w)
               : "l"(p));
}

// Steps that one pass of the sweep handles together (see the comment at the top of the file).
constexpr int PS = 3;

template <int R_, int BP_, bool PROJ, bool PACK, bool META>
__global__ void __launch_bounds__(NT, 1) rollout_bwd_kernel(const BwdArgs a) {
  constexpr int QW = PACK ? 4 : BP_;       // 32-bit words per Q row
  constexpr int QV = QW / 4;               // 16-byte words per Q row
  constexpr int NBX = PACK ? 5 : BP_;      // batch rows the tape and dense loops cover (packed rows: exactly 5)
  // Gather: LPS lanes share a synapse, one per step of the pass (raw rows of four channels: two per
  // step, each taking two channels); the rows they read lie in one or two adjacent lines.
  constexpr int H = (!PROJ && R_ == 4) ? 2 : 1;
  constexpr int LPS = PS * H;
  constexpr int SPG = 32 / LPS;            // synapses per 32-lane group (10 or 5; the last two lanes idle)
  constexpr int CPL = PROJ ? 1 : R_ / H;   // Q rows a lane reads per synapse
  constexpr int QVL = QV * CPL;            // 16-byte words a lane reads per synapse
  constexpr int UF = QVL == 1 ? V1G_BWD_GROUPS : QVL == 2 ? V1G_BWD_GROUPS2 : QVL == 4 ? 2 : 1;  // groups per pass
  constexpr int SPP = SPG * UF;            // synapses per pass
  static_assert(UF <= 4 || PROJ, "the synapse types of a raw pass are kept as four 8-bit fields of one word");
  static_assert(V1G_ROW_PAD % SPG == 0, "padded rows end with a group");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int B = a.B, K = a.K, N = a.N, chunkP = a.chunkP, T = a.T, C = a.C, D = a.D;
  const int n0 = blockIdx.x * a.chunk;
  const int cn = min(a.chunk, N - n0);
  const int nb = B * a.n_bkg;
  auto slot_of = [&](int step) { return (unsigned)((step + K) % K); };  // step >= -K
  // index of a Q row in units of QW words
  auto unit_of = [&](unsigned post, unsigned c, unsigned slot) -> unsigned {
    return PROJ ? (post * (unsigned)C + c) * (unsigned)K + slot : (post * (unsigned)K + slot) * (unsigned)R_ + c;
  };

  unsigned char* sp_ = smem_raw;
  auto take = [&](size_t bytes) {
    unsigned char* p = sp_;
    sp_ += (bytes + 15) & ~(size_t)15;
    return p;
  };
  const size_t plane = (size_t)B * chunkP;
  float* basis_s = (float*)take(sizeof(float) * a.S * R_);
  // per-step planes of a pass, [q][b][k] for step (newest - q)
  float* gz_s = (float*)take(sizeof(float) * PS * plane);  // gathered spike gradient
  float* tv_s = (float*)take(a.tape_in_smem ? sizeof(float) * PS * plane : 0);  // saved words
  float* s_cnt = (float*)take(sizeof(float) * PS * nb);    // background counts of the steps published in the pass
  int* s_misc = (int*)take(sizeof(int) * 8);  // [1] abort flag, [2] rows queued, [4] next queue slot
  unsigned long long* s_ph = (unsigned long long*)take(sizeof(unsigned long long) * 4);  // phase times: tape + wait, gather, dense, end of the last
  // rows to walk in the pass: {first synapse, end, row, spike masks of the steps, 8 bits each}
  int4* rowd_s = (int4*)take(sizeof(int4) * chunkP);
  int* bkptr_s = (int*)take(sizeof(int) * (chunkP + 1));  // background in-synapse ranges, slice-relative
  // background in-synapses of the slice and their weight-gradient accumulators; on chip when they
  // fit, otherwise the global tables are used directly
  int* bk_pre_s = nullptr;
  uint8_t* bk_sid_s = nullptr;
  float* bk_dw_s = nullptr;
  if (a.bkg_in_smem) {
    bk_pre_s = (int*)take(sizeof(int) * a.bkg_cap);
    bk_dw_s = (float*)take(sizeof(float) * a.bkg_cap);
    bk_sid_s = (uint8_t*)take(a.bkg_cap);
  }
  float* base;
  if (a.state_in_smem)
    base = (float*)take(sizeof(float) * plane * (1 + 2 * R_));
  else
    base = a.state_ws + (size_t)blockIdx.x * plane * (1 + 2 * R_);
  float* G_v = base;
  float* G_p = G_v + plane;        // [r][b][k]
  float* G_pr = G_p + plane * R_;  // [r][b][k]

  for (int i = tid; i < a.S * R_; i += NT) basis_s[i] = a.basis[i];
  const int bk_base = a.bkg_inptr[n0];
  const int bk_m = a.bkg_inptr[n0 + cn] - bk_base;
  for (int k = tid; k <= cn; k += NT) bkptr_s[k] = a.bkg_inptr[n0 + k] - bk_base;
  const int* bk_pre = a.bkg_inpre + bk_base;
  const uint8_t* bk_sid = a.bkg_insid + bk_base;
  float* bk_dw = a.dw_bkg + bk_base;
  if (a.bkg_in_smem) {
    for (int j = tid; j < bk_m; j += NT) {
      bk_pre_s[j] = bk_pre[j];
      bk_sid_s[j] = bk_sid[j];
      bk_dw_s[j] = 0.f;
    }
    bk_pre = bk_pre_s;
    bk_sid = bk_sid_s;
    bk_dw = bk_dw_s;
  }
  for (int i = tid; i < (int)plane * (1 + 2 * R_); i += NT) base[i] = 0.f;
  for (int i = tid; i < PS * (int)plane; i += NT) gz_s[i] = 0.f;
  if (tid < 8) s_misc[tid] = 0;
  __syncthreads();
  // phase 0 has nothing to publish (nobody waits for it), but the rotating counters count it
  if (tid == BAR_TID) v1g_arrive(v1g_phase_counter(a.barrier, 0));

  const unsigned long long G = gridDim.x;
  bool ok = true;
  float volt_loss = 0.f;
  // event counts of this thread, added to the 64-bit counters before they can overflow
  unsigned c_rows = 0, c_events = 0, c_dw = 0;
  auto flush_counts = [&]() {
    V1GCounters* c = (V1GCounters*)a.counters;
    const unsigned long long rows = v1g_warp_sum(c_rows), events = v1g_warp_sum(c_events), dw = v1g_warp_sum(c_dw);
    if (lane == 0) {
      if (rows) atomicAdd(&c->bwd_rows, rows);
      if (events) atomicAdd(&c->bwd_events, events);
      if (dw) atomicAdd(&c->dw_events, dw);
    }
    c_rows = c_events = c_dw = 0;
  };
  const bool prof = a.phase_ns != nullptr && tid == 0;
  const unsigned long long ph_start = prof ? gtime_b() : 0;
  if (prof) {
    s_ph[0] = s_ph[1] = s_ph[2] = 0;
    s_ph[3] = ph_start;
  }
  auto lap = [&](int phase) {
    if (prof) {
      const unsigned long long now = gtime_b();
      s_ph[phase] += now - s_ph[3];
      s_ph[3] = now;
    }
  };
  // LGN events are dealt out block by block (event i to block i mod grid), so that every block carries
  // its share of a step's few hundred events
  const int gw = warp * gridDim.x + blockIdx.x, gnw = gridDim.x * NW;

  // Weight gradient of the LGN events of step tt from Q(tt).  One warp per event; the (up to 128)
  // synapses of a pass are loaded together so that the three dependent accesses (record, Q row,
  // atomic) are each paid once per pass.
  auto lgn_dw = [&](int tt) {
    const int seg_per_t = B * a.lgn_nseg;
    const int e0 = a.lgn_off[(int64_t)tt * seg_per_t], e1 = a.lgn_off[(int64_t)(tt + 1) * seg_per_t];
    const unsigned slot = slot_of(tt);
    constexpr int UL = 4;
    for (int e = e0 + gw; e < e1; e += gnw) {
      const uint4 ent = a.lgn_ent4[e];
      const int b = ent.x >> 24;
      const int j0 = (int)ent.y, j1 = (int)ent.z;
      for (int jb = j0; jb < j1; jb += 32 * UL) {
        int post[UL], sid[UL];
#pragma unroll
        for (int q = 0; q < UL; ++q) {
          const int j = jb + q * 32 + lane;
          post[q] = j < j1 ? a.lgn_post[j] : 0;
          sid[q] = j < j1 ? (int)a.lgn_sid[j] : 0;
        }
        float val[UL];
        if (PROJ) {
          float qv[UL][BP_];
#pragma unroll
          for (int q = 0; q < UL; ++q) load_row<BP_, PACK>(a.Q + (size_t)unit_of(post[q], sid[q], slot) * QW, qv[q]);
#pragma unroll
          for (int q = 0; q < UL; ++q) {
            val[q] = 0.f;
#pragma unroll
            for (int bb = 0; bb < BP_; ++bb) val[q] = (bb == b) ? qv[q][bb] : val[q];
          }
        } else {
#pragma unroll
          for (int q = 0; q < UL; ++q) {
            val[q] = 0.f;
#pragma unroll
            for (int r = 0; r < R_; ++r) {
              float qr[BP_];
              load_row<BP_, PACK>(a.Q + (size_t)unit_of(post[q], r, slot) * QW, qr);
              float qb = 0.f;
#pragma unroll
              for (int bb = 0; bb < BP_; ++bb) qb = (bb == b) ? qr[bb] : qb;
              val[q] += qb * basis_s[sid[q] * R_ + r];
            }
          }
        }
#pragma unroll
        for (int q = 0; q < UL; ++q) {
          const int j = jb + q * 32 + lane;
          if (j < j1) atomicAdd(a.dw_lgn + j, val[q]);
        }
      }
      if (lane == 0) c_dw += (unsigned)(j1 - j0);
    }
  };

  // Tape of the steps tn, tn-1, tn-2 into the planes, the rows that must be walked for at least one of them
  // into the queue, and the background counts of the steps tn-2 .. tn-4 that the pass publishes.
  auto load_pass_tape = [&](int tn) {
    for (int k0 = 0; k0 < cn; k0 += NT) {
      const int k = k0 + tid;
      const bool act = k < cn;
      const int n = n0 + (act ? k : 0);
      int rj0 = 0, rj1 = 0;  // the records to walk
      if (act) {
        rj0 = META ? a.rec_brow[n] * V1G_ROW_PAD : a.rec_rowptr[(int64_t)n * D];
        rj1 = META ? a.rec_brow[n + 1] * V1G_ROW_PAD : a.rec_rowptr[(int64_t)n * D + D];
      }
      // all tape loads of the neuron are issued before any of them is used; the word is the voltage with its
      // two lowest mantissa bits = (spiked, refractory)
      unsigned ww[PS][NBX];
#pragma unroll
      for (int q = 0; q < PS; ++q)
#pragma unroll
        for (int b = 0; b < NBX; ++b)
          ww[q][b] = (b < B && act && tn - q >= 0)
                         ? __float_as_uint(__ldcs(a.tape_v + ((int64_t)(tn - q) * B + b) * N + n)) : 2u;
      unsigned live = 0, zm = 0;
#pragma unroll
      for (int q = 0; q < PS; ++q) {
        unsigned z1 = 0, need = 0;
#pragma unroll
        for (int b = 0; b < NBX; ++b) {
          if (b < B && act) {
            if (a.tape_in_smem) tv_s[(q * B + b) * chunkP + k] = __uint_as_float(ww[q][b]);
            z1 |= (ww[q][b] & 1u) << b;
            if (!(ww[q][b] & 2u) && pseudo_h(__uint_as_float(ww[q][b] & ~3u) - 1.f, a) != 0.f) need = 1;
          }
        }
        if (need | z1) live |= 1u << q;
        zm |= z1 << (8 * q);
      }
      // A row is walked when one of the steps has a non-zero pseudo-derivative or a spike.  The planes keep an
      // old value for the others, which the dense part multiplies by a pseudo-derivative of exactly zero.
      const bool walk = live != 0 && rj1 > rj0;
      const unsigned wm = __ballot_sync(0xffffffffu, walk);
      if (wm) {
        int q0 = 0;
        if (lane == 0) q0 = atomicAdd(s_misc + 2, __popc(wm));  // one shared-memory atomic per warp
        q0 = __shfl_sync(0xffffffffu, q0, 0);
        if (walk) {
          rowd_s[q0 + __popc(wm & ((1u << lane) - 1u))] = make_int4(rj0, rj1, k, (int)zm);
          const int len = META ? a.rec_rowptr[(int64_t)n * D + D] - a.rec_rowptr[(int64_t)n * D] : rj1 - rj0;
          c_rows += (unsigned)(D * __popc(live));
          c_events += (unsigned)(len * __popc(live));
          c_dw += (unsigned)(len * __popc(zm));
        }
      }
    }
#pragma unroll
    for (int q = 0; q < PS; ++q)
      if (tn - q >= 2)
        for (int i = tid; i < nb; i += NT) {
          const int b = i / a.n_bkg, j = i - b * a.n_bkg;
          s_cnt[q * nb + i] = (float)a.bkg_counts[((int64_t)b * T + (tn - q - 2)) * a.n_bkg + j];
        }
  };

  // lane's place in the gather: synapse of the group, step of the pass (newest - lq), first of its channels
  const bool lane_on = lane < SPG * LPS;
  const int lsyn = min(lane / LPS, SPG - 1), lrem = lane % LPS;  // idle lanes repeat rows of the last synapse
  const int lq = lrem / H, lch = (lrem % H) * CPL;

  const int n_pass = (T + PS - 1) / PS;
  if (T >= 1) load_pass_tape(T - 1);
  for (int it = 0; it < n_pass && ok; ++it) {
    const int tn = T - 1 - PS * it;  // newest step of the pass
    if (it >= 1) {
      load_pass_tape(tn);
      // LGN weight gradients one pass late: Q of the steps tn+4 .. tn+2 is complete since the previous
      // wait, so this work fills the time that the slowest block still needs
      if (it >= 2)
        for (int q = 4; q >= 2; --q) lgn_dw(tn + q);
      if (tid == BAR_TID) {
        const unsigned long long target = v1g_phase_target(it, G);
        if (v1g_wait(v1g_phase_counter(a.barrier, it), target, a.spin_limit, a.status) < target) s_misc[1] = 1;
      }
    }
    __syncthreads();
    if (s_misc[1]) {
      ok = false;
      break;
    }
    lap(0);

    // ---------------- gather of the pass over the out-synapses of every queued row ----------------
    {
      constexpr int NS = V1G_BWD_STAGES;
      constexpr int NB = NBX;
      struct Rec { unsigned x, y, z; };      // padded record {x, weight}; plain arrays: {post, weight, type | (delay - 1) << 8}
      struct Pass { int jb, j1, k, fl; unsigned zm; };  // fl: 1 first pass of its row, 4 valid
      const int nq = s_misc[2];
      const int jmax = a.rec_nnz - 1;
      const unsigned sb = slot_of(tn - lq + 1);   // slot of this lane's step for a synapse of delay 1
      // Where lanes without a synapse read: a row of the block's own.  One row for the whole grid (row 0) put
      // several requests per walked row on a single L2 slice, which then set the pace (gather 26.3 -> 21.3 us per step).
      const unsigned idle_unit = unit_of((unsigned)n0, 0u, 0u);
      Pass pr{0, 0, 0, 0, 0u};
      Pass ps_[NS];
      Rec rec[UF];
      float4 qS[NS][UF][QVL];
      float wS[NS][UF][CPL];
      unsigned sidS[PROJ ? 1 : NS];  // raw mode: the synapse types of the pass, 8 bits per group (for the weight gradient)
      float acc[NB];
#pragma unroll
      for (int i = 0; i < NS; ++i) ps_[i] = Pass{0, 0, 0, 0, 0u};
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[b] = 0.f;
      auto issue_rec = [&]() {  // advance pr to the following pass and request its records
        if (pr.fl && pr.jb + SPP < pr.j1) {
          pr.jb += SPP;
          pr.fl = 4;
        } else {
          int q = 0;   // warps take rows from the queue one at a time, so a warp that drew long rows takes fewer
          if (lane == 0) q = atomicAdd(s_misc + 4, 1);
          q = __shfl_sync(0xffffffffu, q, 0);
          if (q < nq) {
            const int4 d = rowd_s[q];
            pr = Pass{d.x, d.y, d.z, 5, (unsigned)d.w};
          } else {
            pr = Pass{0, 0, 0, 0, 0u};
          }
        }
#pragma unroll
        for (int u = 0; u < UF; ++u) {
          if (META) {  // whole groups: records past a row's end are the next row's (or the padding of the table)
            const uint2 r = __ldcs(a.rec_pad + pr.jb + u * SPG + lsyn);
            rec[u] = Rec{r.x, r.y, 0u};
          } else {
            const int j = min(pr.jb + u * SPG + lsyn, jmax);
            const int32_t* rp = a.rec_rowptr + (int64_t)(n0 + pr.k) * D;
            unsigned dm1 = 0;
            for (int q = 1; q < D; ++q) dm1 += j >= rp[q] ? 1u : 0u;
            rec[u] = Rec{(unsigned)a.rec_post[j], __float_as_uint(a.rec_w[j]), (unsigned)a.rec_sid[j] | (dm1 << 8)};
          }
        }
      };
      auto issue_q = [&](const Pass& ps, float4 (&q)[UF][QVL], float (&w)[UF][CPL], unsigned& sids) {
        if (!PROJ) sids = 0u;
#pragma unroll
        for (int u = 0; u < UF; ++u) {
          // rows of padded records end with a group, so the test is the same for all lanes
          const bool in_row = META ? ps.jb + u * SPG < ps.j1 : ps.jb + u * SPG + lsyn < ps.j1;
          const unsigned sid = META ? (rec[u].x >> 22) & 127u : rec[u].z & 255u;
          unsigned slot = sb + (META ? rec[u].x >> 29 : rec[u].z >> 8);
          slot = min(slot, slot - (unsigned)K);
          unsigned unit;
          if (PROJ && META)
            unit = (rec[u].x & 0x1fffffffu) * (unsigned)K + slot;
          else
            unit = unit_of(META ? rec[u].x & 0x3fffffu : rec[u].x, PROJ ? sid : (unsigned)lch, slot);
          unit = in_row ? unit : idle_unit;  // what is past the end of the row shares one request
          const float* qp = a.Q + (size_t)(unit * (unsigned)QW);  // < 2^31 words, checked by the host
          // 256-bit loads where every lane's rows start on a 32-byte boundary: 32-byte rows, or an even number
          // of channels per lane (five channels of 16 bytes start on either)
          if (QV == 2 || CPL % 2 == 0) {
#pragma unroll
            for (int v = 0; v + 1 < QVL; v += 2) load_pair(qp + 4 * v, q[u][v], q[u][v + 1]);
          } else {
#pragma unroll
            for (int v = 0; v < QVL; ++v) q[u][v] = __ldcg((const float4*)qp + v);
          }
          const float wt = in_row ? __uint_as_float(rec[u].y) : 0.f;  // the sums of the idle lanes are never read
#pragma unroll
          for (int c = 0; c < CPL; ++c) w[u][c] = PROJ ? wt : wt * basis_s[sid * R_ + lch + c];
          if (!PROJ) sids |= sid << (8 * u);
        }
      };
      auto row_values = [&](const float4 (&q)[QVL], int c, float (&pj)[BP_]) {
        float4 one[PACK ? 1 : BP_ / 4];
#pragma unroll
        for (int v = 0; v < QV; ++v) one[v] = q[c * QV + v];
        unpack_row<BP_, PACK>(one, pj);
      };
      auto reduce_store = [&](int k) {
        // total over the synapse groups: lanes 0 .. LPS-1 end with the sums of their step
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          if (b < B) {
            float v = acc[b];
            if (H == 2) {
              v += __shfl_xor_sync(0xffffffffu, v, 1);
              const float g4 = __shfl_down_sync(0xffffffffu, v, 24);
              v += __shfl_down_sync(0xffffffffu, v, 12);
              v += __shfl_down_sync(0xffffffffu, v, 6);
              v += g4;
            } else {
              v += __shfl_down_sync(0xffffffffu, v, 15);
              const float g4 = __shfl_down_sync(0xffffffffu, v, 12);
              v += __shfl_down_sync(0xffffffffu, v, 6);
              v += __shfl_down_sync(0xffffffffu, v, 3);
              v += g4;
            }
            if (lane < LPS && lane % H == 0) gz_s[(lq * B + b) * chunkP + k] = v;
          }
        }
      };
      auto compute = [&](const Pass& ps, const float4 (&q)[UF][QVL], const float (&w)[UF][CPL], unsigned sids) {
        if (ps.fl & 1) {
#pragma unroll
          for (int b = 0; b < NB; ++b) acc[b] = 0.f;
        }
        if (!ps.zm) {
#pragma unroll
          for (int u = 0; u < UF; ++u) {
#pragma unroll
            for (int c = 0; c < CPL; ++c) {
              float pj[BP_];
              row_values(q[u], c, pj);
#pragma unroll
              for (int b = 0; b < NB; ++b) acc[b] += w[u][c] * pj[b];
            }
          }
        } else {
          // The source neuron spiked in the pass: weight gradient, summed over the lanes (steps) of a synapse.
          // The old values are requested together (a load after a store to the same array would wait for its
          // own round trip); the first lane of a synapse is its only writer.
          const unsigned zq = (ps.zm >> (8 * lq)) & 255u;
          const int nrow = n0 + ps.k;
          const int jo = META ? a.rec_rowptr[(int64_t)nrow * D] - a.rec_brow[nrow] * V1G_ROW_PAD : 0;
          const int j1 = META ? a.rec_rowptr[(int64_t)nrow * D + D] : ps.j1;
          const bool writer = lane_on && lrem == 0;
          float dw_old[UF];
#pragma unroll
          for (int u = 0; u < UF; ++u) {
            const int j = ps.jb + u * SPG + lsyn + jo;
            dw_old[u] = (writer && j < j1) ? a.dw_rec[j] : 0.f;
          }
#pragma unroll
          for (int u = 0; u < UF; ++u) {
            float dwv = 0.f;
#pragma unroll
            for (int c = 0; c < CPL; ++c) {
              float pj[BP_];
              row_values(q[u], c, pj);
              float dws = 0.f;
#pragma unroll
              for (int b = 0; b < NB; ++b) {
                acc[b] += w[u][c] * pj[b];
                if (zq & (1u << b)) dws += pj[b];
              }
              dwv += PROJ ? dws : dws * basis_s[((sids >> (8 * u)) & 255u) * R_ + lch + c];
            }
            if (H == 2) dwv += __shfl_xor_sync(0xffffffffu, dwv, 1);
            dwv += __shfl_down_sync(0xffffffffu, dwv, H) + __shfl_down_sync(0xffffffffu, dwv, 2 * H);
            const int j = ps.jb + u * SPG + lsyn + jo;
            if (writer && j < j1) a.dw_rec[j] = dw_old[u] + dwv;
          }
        }
        if (ps.jb + SPP >= ps.j1) reduce_store(ps.k);
      };
      // One turn of the pipeline with buffer I: false when the warp has no further pass.  Registers that
      // receive a load are never copied while the load is in flight (a copy would wait for it): the loop body
      // is written out once per buffer.
      auto turn = [&](auto I) -> bool {
        constexpr int i = decltype(I)::value;
        if (!pr.fl) {
          // accumulate what is still in flight, oldest first
#pragma unroll
          for (int o = 1; o < NS; ++o)
            if (ps_[(i + o) % NS].fl)
              compute(ps_[(i + o) % NS], qS[(i + o) % NS], wS[(i + o) % NS], sidS[PROJ ? 0 : (i + o) % NS]);
          return false;
        }
        ps_[i] = pr;
        issue_q(ps_[i], qS[i], wS[i], sidS[PROJ ? 0 : i]);
        issue_rec();
        constexpr int x = (i + 1) % NS;  // the oldest pass
        if (ps_[x].fl) {
          compute(ps_[x], qS[x], wS[x], sidS[PROJ ? 0 : x]);
          ps_[x].fl = 0;
        }
        return true;
      };
      issue_rec();
      for (;;) {
        if (!turn(std::integral_constant<int, 0>{})) break;
        if (!turn(std::integral_constant<int, 1 % NS>{})) break;
        if (NS > 2 && !turn(std::integral_constant<int, 2 % NS>{})) break;
      }
    }
    __syncthreads();
    lap(1);
    if (tid == 0) s_misc[2] = s_misc[4] = 0;

    // ------- dense adjoint of the steps of the pass, newest first; publish Q two steps behind; background weight gradient -------
    for (int k = tid; k < cn; k += NT) {
      const int n = n0 + k;
      const float k_decay = a.decay[n] * a.vd_keep, k_cf = a.cf[n];
      const float rcn = a.rate_coef ? a.rate_coef[n] : 0.f;
      const float vlo = a.v_lo ? a.v_lo[n] : 0.f;
#pragma unroll 1
      for (int q = 0; q < PS; ++q) {
        const int t = tn - q;
        if (t < 0) break;
        const float rc = (t >= a.rate_t0 && t < a.rate_t1) ? rcn : 0.f;
        const int bin = (a.sgrad && a.sync_bin > 0 && t / a.sync_bin < a.nbins) ? t / a.sync_bin : -1;
        float gzx[NBX], gvx[NBX];  // loss gradients that do not come from the network: dL/dz and dL/dv
#pragma unroll
        for (int b = 0; b < NBX; ++b) {
          const int64_t oi = ((int64_t)b * T + t) * N + n;
          gzx[b] = (a.g_z && b < B) ? a.g_z[oi] : 0.f;
          gvx[b] = (a.g_v && b < B) ? a.g_v[oi] : 0.f;
        }
        if (bin >= 0) {
#pragma unroll
          for (int b = 0; b < NBX; ++b)
            if (b < B) gzx[b] += a.sgrad[b * a.nbins + bin];
        }
        if (a.sync.first != nullptr && t >= a.sync.t0 && t < a.sync.t0 + a.sync.W) {
          for (int s1 = a.sync.first[n]; s1 >= 0; s1 = a.sync.next[s1]) {
            const int smp = a.sync.pos_sample[s1];
            const int tb = a.sync.trial[smp];
            const float gs = a.sync.g[(int64_t)smp * a.sync.W + (t - a.sync.t0)];
#pragma unroll
            for (int b = 0; b < NBX; ++b) gzx[b] += (b == tb) ? gs : 0.f;
          }
        }
        if (a.osi_coef != nullptr && t >= a.osi_t0 && t < a.osi_t1) {
#pragma unroll
          for (int b = 0; b < NBX; ++b)
            if (b < B) gzx[b] += a.osi_coef[(int64_t)b * N + n];
        }
        float dyv[NBX][R_];  // dy(t-2) of every batch row of this neuron
        // The state of a batch row is read before any of it is written back: a load may not pass an earlier
        // store to the same array, and in a global slab each read would wait an L2 round trip of its own.
#pragma unroll
        for (int b = 0; b < NBX; ++b) {
#pragma unroll
          for (int r = 0; r < R_; ++r) dyv[b][r] = 0.f;
          if (b < B) {
            const float sv = G_v[b * chunkP + k];
            float sp[R_], spr[R_];
#pragma unroll
            for (int r = 0; r < R_; ++r) {
              sp[r] = G_p[(r * B + b) * chunkP + k];
              spr[r] = G_pr[(r * B + b) * chunkP + k];
            }
            const int pi = (q * B + b) * chunkP + k;
            const unsigned word = __float_as_uint(a.tape_in_smem ? tv_s[pi] : a.tape_v[((int64_t)t * B + b) * N + n]);
            const float v = __uint_as_float(word & ~3u);
            const bool free_ = !(word & 2u);
            const float gz = rc + gzx[b] + a.rec_factor * gz_s[pi];
            float gv = sv + gvx[b];
            if (a.volt_coef != 0.f) {
              // range mode: outside [vlo, 1]; threshold mode: distance from the threshold
              const float hi = a.volt_threshold_mode ? v - 1.f : fmaxf(v - 1.f, 0.f);
              const float lo = a.volt_threshold_mode ? 0.f : fmaxf(vlo - v, 0.f);
              gv += 2.f * a.volt_coef * (hi - lo);
              volt_loss += hi * hi + lo * lo;
            }
            if (free_) gv += gz * pseudo_h(v - 1.f, a);
            if (a.hard_reset && !free_) gv = 0.f;
            G_v[b * chunkP + k] = k_decay * gv;
            const float gc1 = k_cf * gv;
#pragma unroll
            for (int r = 0; r < R_; ++r) {
              const float gp1 = a.sd[r] * sp[r] + gc1;                   // g_p(t-1)
              const float gpr1 = a.sd[r] * spr[r] + a.dtsd[r] * sp[r];   // g_pr(t-1)
              G_p[(r * B + b) * chunkP + k] = gp1;
              G_pr[(r * B + b) * chunkP + k] = gpr1;
              const float gpr2 = a.sd[r] * gpr1 + a.dtsd[r] * gp1;       // g_pr(t-2)
              dyv[b][r] = (gpr2 * a.pinit[r]) * a.lr_scale;
            }
          }
        }
        if (t >= 2) {
          // one 16/32-byte row per channel, all batch rows of the neuron at once
          const unsigned slot = slot_of(t - 2);
          for (int c = 0; c < C; ++c) {
            float row[NBX];
#pragma unroll
            for (int b = 0; b < NBX; ++b) {
              float s2 = 0.f;
              if (PROJ) {
#pragma unroll
                for (int r = 0; r < R_; ++r) s2 += basis_s[c * R_ + r] * dyv[b][r];
              } else {
#pragma unroll
                for (int r = 0; r < R_; ++r) s2 = (r == c) ? dyv[b][r] : s2;
              }
              row[b] = s2;
            }
            float4* qd = (float4*)(a.Q + (size_t)unit_of((unsigned)n, (unsigned)c, slot) * QW);
            if (PACK) {
              float r8[8];
#pragma unroll
              for (int b = 0; b < 8; ++b) r8[b] = b < NBX ? row[b % NBX] : 0.f;
              __stcg(qd, pack_row5(r8));
            } else {
              __stcg(qd, make_float4(row[0], row[1], row[2], row[3]));
              if (BP_ == 8) __stcg(qd + 1, make_float4(row[4 % NBX], row[5 % NBX], row[6 % NBX], row[7 % NBX]));
            }
          }
          // background weight gradient of step t-2 for the synapses this thread owns (branch-free:
          // a zero count contributes zero)
          const float* cnt = s_cnt + q * nb;
          auto bkg_grad = [&](int pre, int sid) {
            const float* bs = basis_s + sid * R_;
            float bsr[R_];
#pragma unroll
            for (int r = 0; r < R_; ++r) bsr[r] = bs[r];
            float accw = 0.f;
#pragma unroll
            for (int b = 0; b < NBX; ++b) {
              if (b < B) {
                float s2 = 0.f;
#pragma unroll
                for (int r = 0; r < R_; ++r) s2 += dyv[b][r] * bsr[r];
                accw += s2 * cnt[b * a.n_bkg + pre];
              }
            }
            return accw;
          };
          if (a.bkg_in_smem) {
            for (int j = bkptr_s[k]; j < bkptr_s[k + 1]; ++j) bk_dw[j] += bkg_grad(bk_pre[j], (int)bk_sid[j]);
          } else {
            // tables and accumulators in global memory: four synapses' entries are requested together
            for (int j0 = bkptr_s[k], j1 = bkptr_s[k + 1]; j0 < j1; j0 += 4) {
              int pre[4], sid[4];
              float old[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int j = min(j0 + u, j1 - 1);
                pre[u] = bk_pre[j];
                sid[u] = (int)bk_sid[j];
                old[u] = bk_dw[j];
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const float accw = bkg_grad(pre[u], sid[u]);
                if (j0 + u < j1 && accw != 0.f) bk_dw[j0 + u] = old[u] + accw;
              }
            }
          }
        }
      }
    }
    __syncthreads();
    if (tid == BAR_TID) v1g_arrive(v1g_phase_counter(a.barrier, it + 1));
    lap(2);
    if (__any_sync(0xffffffffu, ((c_rows | c_events | c_dw) >> 30) != 0)) flush_counts();
  }
  // ---- full barrier: Q(0..D-1) of every block is in the ring ----
  if (tid == BAR_TID && ok && n_pass >= 1) {
    const unsigned long long target = v1g_phase_target(n_pass, G);
    if (v1g_wait(v1g_phase_counter(a.barrier, n_pass), target, a.spin_limit, a.status) < target) s_misc[1] = 1;
  }
  __syncthreads();
  ok = ok && !s_misc[1];
  // LGN weight gradients of the steps that the loop has not reached (it runs one pass behind)
  if (ok)
    for (int tt = min(T - 1 - PS * (n_pass - 1) + 1, T - 3); tt >= 0; --tt) lgn_dw(tt);
  // Spikes that were pending in the initial z_buf (emitted at step -(kb+1), bit kb) are delivered
  // at steps 0..D-1 and contribute to the recurrent weight gradient; Q(0..D-1) is still in the ring.
  if (ok && a.hist0) {
    for (int k = warp; k < cn; k += NW) {
      const int32_t* rp = a.rec_rowptr + (int64_t)(n0 + k) * D;
      const int j0 = rp[0], j1 = rp[D];
      for (int b = 0; b < B; ++b) {
        const unsigned hbits = a.hist0[(int64_t)b * N + n0 + k];
        if (!hbits) continue;
        for (int j = j0 + lane; j < j1; j += 32) {
          int d = 1;
          for (int q = 1; q < D; ++q) d += (j >= rp[q]) ? 1 : 0;
          const int post = a.rec_post[j], sid = a.rec_sid[j];
          float dwv = 0.f;
          for (int kb = 0; kb < D; ++kb) {
            const int sstep = d - (kb + 1);
            if (!(hbits & (1u << kb)) || sstep < 0 || sstep >= T) continue;
            const unsigned slot = slot_of(sstep);
            float pj[BP_];
            if (PROJ) {
              load_row<BP_, PACK>(a.Q + (size_t)unit_of(post, sid, slot) * QW, pj);
            } else {
#pragma unroll
              for (int bb = 0; bb < BP_; ++bb) pj[bb] = 0.f;
#pragma unroll
              for (int r = 0; r < R_; ++r) {
                float q[BP_];
                load_row<BP_, PACK>(a.Q + (size_t)unit_of(post, r, slot) * QW, q);
#pragma unroll
                for (int bb = 0; bb < BP_; ++bb) pj[bb] += q[bb] * basis_s[sid * R_ + r];
              }
            }
#pragma unroll
            for (int bb = 0; bb < BP_; ++bb) dwv += (bb == b) ? pj[bb] : 0.f;
          }
          if (dwv != 0.f) a.dw_rec[j] += dwv;
        }
      }
    }
  }
  if (a.bkg_in_smem)
    for (int j = tid; j < bk_m; j += NT) a.dw_bkg[bk_base + j] += bk_dw_s[j];

  if (prof) {
    unsigned long long* o = a.phase_ns + 4 * blockIdx.x;
    o[0] = s_ph[2];  // dense adjoint
    o[1] = s_ph[1];  // gather
    o[2] = s_ph[0];  // wait + tape
    o[3] = gtime_b() - ph_start;
  }
  // voltage loss and counters
  for (int o = 16; o > 0; o >>= 1) volt_loss += __shfl_down_sync(0xffffffffu, volt_loss, o);
  if (lane == 0 && volt_loss != 0.f) atomicAdd(a.loss_acc + 2, volt_loss * a.volt_coef);
  flush_counts();
}

template <int R_, int BP_, bool PROJ, bool PACK, bool META>
int launch_bwd_m(V1GHandle* h, const BwdArgs& a, int grid, size_t smem, cudaStream_t st) {
  auto kern = rollout_bwd_kernel<R_, BP_, PROJ, PACK, META>;
  V1G_CUDA(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  V1G_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem));
  if (per_sm < 1 || grid > per_sm * h->n_sms)
    return v1g_fail(h, V1G_ERANGE, "rollout grid of %d blocks cannot be co-resident (%d per SM)", grid, per_sm);
  void* args[] = {(void*)&a};
  V1G_CUDA(h, cudaEventRecord(h->ev[2], st));
  V1G_CUDA(h, cudaLaunchCooperativeKernel((void*)kern, dim3(grid), dim3(NT), args, smem, st));
  V1G_CUDA(h, cudaEventRecord(h->ev[3], st));
  h->ev_valid[1] = true;
  v1g_count_launches(1);
  return V1G_OK;
}

template <int R_, int BP_, bool PROJ, bool PACK>
int launch_bwd(V1GHandle* h, const BwdArgs& a, int grid, size_t smem, cudaStream_t st) {
  return a.rec_pad ? launch_bwd_m<R_, BP_, PROJ, PACK, true>(h, a, grid, smem, st)
                   : launch_bwd_m<R_, BP_, PROJ, PACK, false>(h, a, grid, smem, st);
}

}  // namespace

// One translation unit per (channels, batch values of a Q row), so that they compile side by side.
int v1g_launch_bwd_r4_b4(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st);
int v1g_launch_bwd_r4_b8(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st);
int v1g_launch_bwd_r5_b4(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st);
int v1g_launch_bwd_r5_b8(V1GHandle* h, const BwdArgs& a, bool proj, bool pack, int grid, size_t smem, cudaStream_t st);
