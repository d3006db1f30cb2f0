// Forward rollout, register-resident variant: one thread per neuron, the batch unrolled at
// compile time, the state of all batch rows of the neuron held on chip for the whole rollout: v, psc,
// refractory counter and spike history in registers, psc_rise and the after-spike currents in
// conflict-free shared-memory planes (see asc_in_smem below for the split).  Per-neuron constants and the neuron's
// background in-synapses are read once per neuron and step instead of once per (batch, neuron).
// Used when the block slice has at most V1G_NT_REG neurons; otherwise the shared-memory kernel in
// v1g_rollout_fwd.cu runs.  Synchronisation, ring protocol and arithmetic (operation order
// included) are identical to that kernel.
#include <algorithm>
#include <type_traits>

#include "v1g_rollout_fwd.cuh"

namespace {

// asynchronous global -> shared copies of 4 and 16 bytes (both addresses aligned to the size)
__device__ __forceinline__ void cp_async_4(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)), "l"(gsrc) : "memory");
}

constexpr int NT = V1G_NT_REG;
constexpr int NW = NT / 32;
// State that a thread touches once per row and step lives in shared memory instead of registers (128 per
// thread): psc_rise always; the after-spike currents up to 6 rows, psc from 7 rows on (both together
// would not fit for 8 rows of 5 channels).  8 rows take 16.5 us per step at 66,634 neurons; the
// shared-memory kernel, which has no registers to spill but walks the rows one after another, took 30.2.
__host__ __device__ constexpr bool asc_in_smem(int B) { return B <= 6; }
__host__ __device__ constexpr bool psc_in_smem(int B) { return B > 6; }

// The dense phase takes two batch rows at a time: sm_100a multiplies and adds two floats per instruction
// (each rounded on its own, so the results are those of the scalar operations), and what the rows
// share - background synapses, basis rows, constants - is read once.  A last odd row goes alone.  The
// dense phase is bound by instruction issue, 15 warps per SM with one neuron per thread; microseconds per
// step one row at a time and in pairs, 66,634 neurons at 4 Hz: batch 5 10.00 -> 9.20, batch 4 7.95 -> 7.50,
// batch 5 with 121 synapse types 12.84 -> 12.72 (there the scatter is as long as the dense phase).
struct f2 {
  unsigned long long x;
};
template <int W> struct RowVec;
template <> struct RowVec<1> { using T = float; };
template <> struct RowVec<2> { using T = f2; };
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d.x) : "f"(lo), "f"(hi));
  return d;
}
// The assembler contracts a packed multiply and a packed add even under -fmad=false, which changes the
// results (a third of the voltages of one step in their last bit).  A product is therefore a multiply-add
// of a minus zero that the compiler cannot know: a * b + (-0) is a * b, rounded once, sign of zero included.
__device__ __forceinline__ f2 mul_nz(f2 a, f2 b, unsigned long long minus_zero) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.x) : "l"(a.x), "l"(b.x), "l"(minus_zero));
  return d;
}
__device__ __forceinline__ f2 add(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.x) : "l"(a.x), "l"(b.x));
  return d;
}
__device__ __forceinline__ f2 sub(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d.x) : "l"(a.x), "l"(b.x));
  return d;
}
__device__ __forceinline__ float mul_nz(float a, float b, unsigned long long) { return a * b; }
__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ float sub(float a, float b) { return a - b; }
template <int W> __device__ __forceinline__ typename RowVec<W>::T all(float v);
template <> __device__ __forceinline__ float all<1>(float v) { return v; }
template <> __device__ __forceinline__ f2 all<2>(float v) { return pack2(v, v); }
// neighbouring rows in shared memory
template <int W> __device__ __forceinline__ typename RowVec<W>::T load_rows(const float* s);
template <> __device__ __forceinline__ float load_rows<1>(const float* s) { return *s; }
template <> __device__ __forceinline__ f2 load_rows<2>(const float* s) { return f2{*reinterpret_cast<const unsigned long long*>(s)}; }
__device__ __forceinline__ void store_rows(float* s, float v) { *s = v; }
__device__ __forceinline__ void store_rows(float* s, f2 v) { *reinterpret_cast<unsigned long long*>(s) = v.x; }
// values of rows b .. b + W - 1 of a per-row array
template <int W> __device__ __forceinline__ typename RowVec<W>::T rows_of(const float* v);
template <> __device__ __forceinline__ float rows_of<1>(const float* v) { return v[0]; }
template <> __device__ __forceinline__ f2 rows_of<2>(const float* v) { return pack2(v[0], v[1]); }
__device__ __forceinline__ void put_rows(float* v, float d) { v[0] = d; }
__device__ __forceinline__ void put_rows(float* v, f2 d) { asm("mov.b64 {%0, %1}, %2;" : "=f"(v[0]), "=f"(v[1]) : "l"(d.x)); }

template <int R_, int B_>
__global__ void __launch_bounds__(NT, 1) rollout_fwd_reg_kernel(const FwdArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int D = a.D, K = a.K, N = a.N, Np = a.Np;
  auto mul = [&](auto x, auto y) { return mul_nz(x, y, a.minus_zero2); };
  // equal slices, or slices of equal scatter work (at most one neuron per thread either way)
  const int n0 = a.slice ? a.slice[blockIdx.x] : blockIdx.x * a.chunk;
  const int cn = a.slice ? a.slice[blockIdx.x + 1] - n0 : min(a.chunk, N - n0);
  const bool active = tid < cn;
  // One thread of the last warp arrives at and waits on the phase counters.  Its release completes only
  // when the block's atomics of the step have been performed, and whatever shares its warp waits with it;
  // the last warp is the one with the fewest neurons (none at up to 480 per block).  5,000 neurons, batch 2:
  // 5.11 us per step with thread 0, 4.40 with the last warp; no difference at 450 neurons per block.
  const bool ctl = tid == NT - 32;
  const int n = n0 + (active ? tid : 0);
  const int nb = B_ * a.n_bkg;
  constexpr int BP = (B_ + 1) & ~1;   // counts are held [node][BP], so that a pair of rows is one load
  constexpr int RQ = (R_ + 1) & ~1;

  unsigned char* sp_ = smem_raw;
  auto take = [&](size_t bytes) {
    unsigned char* p = sp_;
    sp_ += (bytes + 15) & ~(size_t)15;
    return p;
  };
  float* basis_s = (float*)take(sizeof(float) * a.S * R_);
  uint32_t* spk_list = (uint32_t*)take(sizeof(uint32_t) * B_ * NT);
  float2* basis_d = (float2*)take(sizeof(float2) * a.S * RQ);   // every entry twice
  int* s_cnt = (int*)take(sizeof(int) * 2 * BP * a.n_bkg);
  // [1] abort, [2],[3] spike counts by parity, [8 + 2*(s&3)], [9 + 2*(s&3)] bounds of the LGN events of step s
  int* s_misc = (int*)take(sizeof(int) * 16);
  unsigned long long* ctr_s = (unsigned long long*)take(sizeof(unsigned long long) * (4 * NW + 4));
  int2* rowb_s = (int2*)take(sizeof(int2) * NT);   // [first, end) of each neuron's out-synapses
  uint4* lgn_ent_s = (uint4*)take(sizeof(uint4) * 2 * NW);  // per warp: its first LGN event of the next two steps
  uint2* bk_s = (uint2*)take(sizeof(uint2) * a.bkg_cap);  // (pre * BP | sid << 24, weight bits)
  // planes of Q values per row: [pair][Q][tid] of two rows each, then [Q][tid] of an odd last row
  auto plane = [&](float* base, int Q, int b, int r) -> float* {
    return b < (B_ & ~1) ? base + 2 * (((b >> 1) * Q + r) * NT + tid) + (b & 1) : base + ((B_ & ~1) * Q + r) * NT + tid;
  };
  float* pr_s = (float*)take(sizeof(float) * B_ * R_ * NT);
  auto pr_row = [&](int b, int r) { return plane(pr_s, R_, b, r); };
  constexpr bool ASM = asc_in_smem(B_), PSM = psc_in_smem(B_);
  float* as_s = (float*)take(ASM ? sizeof(float) * B_ * 2 * NT : 0);
  float* p_s = (float*)take(PSM ? sizeof(float) * B_ * R_ * NT : 0);
  float as_g[ASM ? 1 : B_][2], p_g[PSM ? 1 : B_][R_];
  auto as_row = [&](int b, int k) -> float* { return ASM ? plane(as_s, 2, b, k) : &as_g[ASM ? 0 : b][k]; };
  auto p_row = [&](int b, int r) -> float* { return PSM ? plane(p_s, R_, b, r) : &p_g[PSM ? 0 : b][r]; };
#define PR(b, r) (*pr_row(b, r))
#define PSC(b, r) (*p_row(b, r))

  for (int i = tid; i < a.S * R_; i += NT) {
    basis_s[i] = a.basis[i];
    basis_d[i / R_ * RQ + i % R_] = make_float2(a.basis[i], a.basis[i]);
  }
  for (int i = tid; i < 2 * BP * a.n_bkg; i += NT) s_cnt[i] = 0;
  const int bk_base = a.bkg_inptr[n0];
  {
    const int m = a.bkg_inptr[n0 + cn] - bk_base;
    for (int j = tid; j < m; j += NT)
      bk_s[j] = make_uint2((uint32_t)(a.bkg_inpre[bk_base + j] * BP) | ((uint32_t)a.bkg_insid[bk_base + j] << 24),
                           __float_as_uint(a.bkg_w[bk_base + j]));
  }
  const int bj0 = active ? a.bkg_inptr[n] - bk_base : 0;
  const int bj1 = active ? a.bkg_inptr[n + 1] - bk_base : 0;
  const float k_decay = a.decay[n], k_cf = a.cf[n];
  const float k_ad0 = a.asc_decay[2 * n], k_ad1 = a.asc_decay[2 * n + 1];
  const float k_am0 = a.asc_amps[2 * n], k_am1 = a.asc_amps[2 * n + 1];
  const int k_tref = a.tref[n];

  // ---- state in registers ----
  float v[B_];
  unsigned rh[B_];  // bits 0..7 spike history (bit d-1 = spiked d steps ago), bits 8..15 refractory
  const bool have_state = a.st.v != nullptr;
#pragma unroll
  for (int b = 0; b < B_; ++b) {
    v[b] = 0.f;
    *as_row(b, 0) = *as_row(b, 1) = 0.f;
    rh[b] = 0;
#pragma unroll
    for (int r = 0; r < R_; ++r) {
      PSC(b, r) = 0.f;
      PR(b, r) = 0.f;
    }
    if (have_state && active) {
      const int64_t g = (int64_t)b * N + n;
      v[b] = a.st.v[g];
      *as_row(b, 0) = a.st.asc[2 * g];
      *as_row(b, 1) = a.st.asc[2 * g + 1];
#pragma unroll
      for (int r = 0; r < R_; ++r) {
        PSC(b, r) = a.st.psc[g * R_ + r];
        PR(b, r) = a.st.psc_rise[g * R_ + r];
      }
      unsigned hist = 0;
      for (int d = 0; d < D; ++d)
        if (a.st.z_buf[((int64_t)b * D + d) * N + n] > 0.f) hist |= 1u << d;
      rh[b] = hist | ((unsigned)(uint8_t)a.st.r[g] << 8);
    }
  }
  if (tid < 16) s_misc[tid] = 0;
  if (tid < 4 * NW + 4) ctr_s[tid] = 0;
  rowb_s[tid] = active ? make_int2(a.rec_rowptr[(int64_t)n * D], a.rec_rowptr[(int64_t)n * D + D]) : make_int2(0, 0);
  __syncthreads();

  // event counters of the warp's lane 0 (in shared memory: the registers are all taken)
  unsigned long long *ctr = ctr_s + 4 * warp, &c_rec_ev = ctr[0], &c_lgn_rows = ctr[1], &c_lgn_ev = ctr[2], &c_spikes = ctr[3];
  // LGN events are dealt out over the grid's warps block by block (event i to block i mod grid), the
  // last warps of a block first: numbered block-major, the few hundred events of a step all fell on
  // the first third of the blocks, which then set the pace of every step
  const int gw = (NW - 1 - warp) * gridDim.x + blockIdx.x, gnw = gridDim.x * NW;

  // ---- prologue: pending deliveries of the initial spike buffer, LGN events of step 0 ----
  if (have_state) {
    // every warp walks the pending spikes of its own lanes, one lane at a time
#pragma unroll
    for (int b = 0; b < B_; ++b) {
      for (int d = 0; d < D; ++d) {
        unsigned m = __ballot_sync(0xffffffffu, active && (rh[b] & (1u << d)));
        while (m) {
          const int src = __ffs(m) - 1;
          m &= m - 1;
          v1g_walk_rec<R_>(a, basis_s, lane, b, a.rec_rowptr + (int64_t)(n0 + warp * 32 + src) * D,
                           -(d + 1), c_rec_ev);
        }
      }
    }
  }
  if (a.T > 0)
    v1g_scatter_lgn<R_>(a, basis_s, lane, gw, gnw, v1g_lgn_begin(a, 0), v1g_lgn_begin(a, 1), 0, c_lgn_rows, c_lgn_ev);
  // LGN hand-over: the bounds of the events of steps 1 and 2, and every warp's first event of step 1
  const bool lgn8 = a.lgn_syn8 != nullptr;
  if (tid == 0) {
    for (int s = 1; s <= 2; ++s) {
      s_misc[8 + 2 * (s & 3)] = s < a.T ? v1g_lgn_begin(a, s) : 0;
      s_misc[9 + 2 * (s & 3)] = s < a.T ? v1g_lgn_begin(a, s + 1) : 0;
    }
  }
  if (lane == 0) {
    uint4 ent = make_uint4(0u, 0u, 0u, 0u);
    if (a.T > 1) {
      const int e = v1g_lgn_begin(a, 1) + gw;
      if (e < v1g_lgn_begin(a, 2)) ent = a.lgn_ent4[e];
    }
    lgn_ent_s[(1 & 1) * NW + warp] = ent;
  }
  __syncthreads();
  if (ctl) v1g_arrive(v1g_phase_counter(a.barrier, 0));

  const unsigned hist_mask = (1u << D) - 1u;
  const unsigned long long G = gridDim.x;
  const bool prof = a.phase_ns != nullptr && tid == 0;
  unsigned long long *ph = ctr_s + 4 * NW, &ph_dense = ph[0], &ph_scatter = ph[1], &ph_barrier = ph[2];
  if (prof) ph[3] = gtime();
  bool seen = false;   // the phase that the next iteration waits for is complete (thread ctl)
  bool ok = true;

  // background input of W batch rows of this neuron: sum over its in-synapses of
  // (w * count) * basis[sid, :] (models.py:890-934 in post-major form)
  auto bkg_gather = [&](auto wc_, int b, const int* cnt_s, auto& Gs) {
    constexpr int W = decltype(wc_)::value;
#pragma unroll
    for (int r = 0; r < R_; ++r) Gs[r] = all<W>(0.f);
    // branch-free: a zero count adds +0 to every channel, which leaves the sums unchanged
    for (int j = bj0; j < bj1; ++j) {
      const uint2 e = bk_s[j];
      const int* cp = cnt_s + (e.x & 0xffffffu) + b;
      if constexpr (W == 2) {
        const int2 cnt = *reinterpret_cast<const int2*>(cp);
        const f2 wc = mul(all<2>(__uint_as_float(e.y)), pack2((float)cnt.x, (float)cnt.y));
        const ulonglong2* bs = reinterpret_cast<const ulonglong2*>(basis_d + (e.x >> 24) * RQ);
#pragma unroll
        for (int r = 0; r < R_; r += 2) {
          const ulonglong2 q = bs[r / 2];
          Gs[r] = add(Gs[r], mul(wc, f2{q.x}));
          if (r + 1 < R_) Gs[r + 1] = add(Gs[r + 1], mul(wc, f2{q.y}));
        }
      } else {
        const int cnt = *cp;
        const float wc = __uint_as_float(e.y) * (float)cnt;
        const float* bs = basis_s + (e.x >> 24) * R_;
#pragma unroll
        for (int r = 0; r < R_; ++r) Gs[r] += wc * bs[r];
      }
    }
  };
  using W1 = std::integral_constant<int, 1>;
  using W2 = std::integral_constant<int, 2>;

  for (int t = 0; t < a.T && ok; ++t) {
    const unsigned long long ph0 = prof ? gtime() : 0;
    if (ctl && t >= 2) {
      const unsigned long long target = v1g_phase_target(t - 2, G);
      if (!seen) seen = v1g_wait(v1g_phase_counter(a.barrier, t - 2), target, a.spin_limit, a.status) >= target;
      if (!seen) s_misc[1] = 1;
    }
    __syncthreads();
    if (s_misc[1]) {
      ok = false;
      break;
    }
    if (ctl && t >= 1) v1g_arrive(v1g_phase_counter(a.barrier, t));
    const unsigned long long ph1 = prof ? gtime() : 0;
    const bool consume = t >= 2;
    const int slot = consume ? (t - 2) % K : 0;
    const int* cnt_s = s_cnt + (t & 1) * BP * a.n_bkg;
    if (t >= 1) {
      // counts of step t-1 for the next iteration, copied asynchronously into the other buffer
      int* cnt_n = s_cnt + ((t + 1) & 1) * BP * a.n_bkg;
      for (int i = tid; i < nb; i += NT) {
        const int b = i / a.n_bkg, j = i - b * a.n_bkg;
        cp_async_4(cnt_n + j * BP + b, a.bkg_counts + ((int64_t)b * a.T + (t - 1)) * a.n_bkg + j);
      }
    }
    int* nspk_p = &s_misc[2 + (t & 1)];

#ifndef V1G_FWD_NO_ROW_PREFETCH
    // the same for the LGN event this warp scatters after the dense phase (fetched an iteration ago)
    if (lane == 0 && lgn8 && t + 1 < a.T) {
      const uint4 ent = lgn_ent_s[((t + 1) & 1) * NW + warp];
      const char* p0 = (const char*)(a.lgn_syn8 + ent.y);
      const char* p1 = (const char*)(a.lgn_syn8 + ent.z);
      for (const char* p = p0; p < p1; p += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
#endif
    // ---------------- dense phase ----------------
    if (active) {
      // ring values of the next rows are requested while these are processed
      float* rp = a.ring + ((int64_t)slot * B_ * R_) * Np + n;
      float Ic[R_][2], In_[R_][2];
      auto request = [&](int b, float (&I)[R_][2]) {
#pragma unroll
        for (int r = 0; r < R_; ++r)
#pragma unroll
          for (int w = 0; w < 2; ++w)
            if (b + w < B_) I[r][w] = __ldcg(rp + (int64_t)((b + w) * R_ + r) * Np);
      };
      if (consume) request(0, Ic);
      auto rows = [&](auto wc_, int b) {
        constexpr int W = decltype(wc_)::value;
        using V = typename RowVec<W>::T;
        V prv[R_];
#pragma unroll
        for (int r = 0; r < R_; ++r) {
          prv[r] = load_rows<W>(pr_row(b, r));
        }
        if (consume) {
          if (b + W < B_) request(b + W, In_);
          V Gs[R_];
          bkg_gather(wc_, b, cnt_s, Gs);
#pragma unroll
          for (int r = 0; r < R_; ++r) {
#pragma unroll
            for (int w = 0; w < W; ++w) __stcg(rp + (int64_t)((b + w) * R_ + r) * Np, 0.f);
            prv[r] = add(mul(prv[r], all<W>(a.sd[r])),
                         mul(mul(add(rows_of<W>(Ic[r]), Gs[r]), all<W>(a.lr_scale)), all<W>(a.pinit[r])));
            store_rows(pr_row(b, r), prv[r]);
            Ic[r][0] = In_[r][0];
            Ic[r][1] = In_[r][1];
          }
        }
        V csum = all<W>(0.f);
#pragma unroll
        for (int r = 0; r < R_; ++r) {
          V pn;
          [[maybe_unused]] float pb[W];
          if constexpr (PSM) {
            pn = load_rows<W>(p_row(b, r));
          } else {
#pragma unroll
            for (int w = 0; w < W; ++w) pb[w] = PSC(b + w, r);
            pn = rows_of<W>(pb);
          }
          if (t >= 1) {
            pn = add(mul(pn, all<W>(a.sd[r])), mul(all<W>(a.dtsd[r]), prv[r]));
            if constexpr (PSM) {
              store_rows(p_row(b, r), pn);
            } else {
              put_rows(pb, pn);
#pragma unroll
              for (int w = 0; w < W; ++w) PSC(b + w, r) = pb[w];
            }
          }
          csum = (r == 0) ? pn : add(csum, pn);
        }
        float pz[W];
#pragma unroll
        for (int w = 0; w < W; ++w) pz[w] = (rh[b + w] & 1u) ? 1.f : 0.f;
        const V prev_z = rows_of<W>(pz);
        V va[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if constexpr (ASM) {
            va[k] = load_rows<W>(as_row(b, k));
          } else {
            float q[W];
#pragma unroll
            for (int w = 0; w < W; ++w) q[w] = *as_row(b + w, k);
            va[k] = rows_of<W>(q);
          }
        }
        const V c1 = add(csum, add(va[0], va[1]));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          va[k] = add(mul(all<W>(k ? k_ad1 : k_ad0), va[k]), mul(prev_z, all<W>(k ? k_am1 : k_am0)));
          if constexpr (ASM) {
            store_rows(as_row(b, k), va[k]);
          } else {
            float q[W];
            put_rows(q, va[k]);
#pragma unroll
            for (int w = 0; w < W; ++w) *as_row(b + w, k) = q[w];
          }
        }
        const V vv = rows_of<W>(v + b);
        const V dv = add(mul(vv, all<W>(a.vd_keep)), mul(vv, all<W>(a.vd_drop)));
        put_rows(v + b, sub(add(mul(all<W>(k_decay), dv), mul(all<W>(k_cf), c1)), prev_z));
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const unsigned hist = rh[b + w] & 0xffu;
          float nv = v[b + w];
          int nr = (int)(rh[b + w] >> 8) + ((hist & 1u) ? k_tref : 0) - 1;
          nr = nr > 0 ? nr : 0;
          if (a.hard_reset && nr > 0) nv = 0.f;
          const bool z = ((nv - 1.f) > 0.f) && (nr == 0);
          v[b + w] = nv;
          rh[b + w] = (((hist << 1) | (z ? 1u : 0u)) & hist_mask) | ((unsigned)nr << 8);
          const int64_t oi = ((int64_t)(b + w) * a.T + t) * N + n;
          if (a.z_out) __stcs(a.z_out + oi, (uint8_t)(z ? 1 : 0));
          if (a.v_out) __stcs(a.v_out + oi, nv);
          if (a.tape_v) {
            const int64_t ti = ((int64_t)t * B_ + b + w) * N + n;
            // the voltage with its two lowest mantissa bits replaced by (spiked, refractory)
            __stcs(a.tape_v + ti, __uint_as_float((__float_as_uint(nv) & ~3u) | (z ? 1u : 0u) | (nr > 0 ? 2u : 0u)));
          }
          if (z) {
            spk_list[atomicAdd(nspk_p, 1)] = ((uint32_t)(b + w) << 24) | (uint32_t)tid;
#ifndef V1G_FWD_NO_ROW_PREFETCH
            // the scatter phase will walk this neuron's out-synapses: ask L2 for their records now, so that
            // they are on their way from HBM while the rest of the dense phase runs
            if (a.rec_syn8) {
              const int2 rb = rowb_s[tid];
              const char* p0 = (const char*)(a.rec_syn8 + rb.x);
              const char* p1 = (const char*)(a.rec_syn8 + rb.y);
              for (const char* q = p0; q < p1; q += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
            }
#endif
          }
        }
      };
#pragma unroll
      for (int b = 0; b + 2 <= B_; b += 2) rows(W2{}, b);
      if constexpr (B_ & 1) rows(W1{}, B_ - 1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const unsigned long long ph2 = prof ? gtime() : 0;
    // ---------------- scatter phase ----------------
    if (ctl) {
      seen = t >= 1 && v1g_ld_acquire(v1g_phase_counter(a.barrier, t - 1)) >= v1g_phase_target(t - 1, G);
      s_misc[2 + ((t + 1) & 1)] = 0;
    }
    const int nspk = *nspk_p;
    for (int e = warp; e < nspk; e += NW) {
      const uint32_t ent = spk_list[e];
      if (a.stat_neuron && lane == 0) {
        atomicAdd(a.stat_neuron + n0 + (int)(ent & 0xffffffu), 1);
        atomicAdd(a.stat_pop + t * B_ + (int)(ent >> 24), 1);
      }
      if (a.rec_syn8) {
        const int2 rb = rowb_s[ent & 0xffffffu];
        v1g_scatter_row8<R_>(a, a.rec_syn8, basis_s, lane, (int)(ent >> 24), rb.x, rb.y, t % K, true);
        if (lane == 0) c_rec_ev += (unsigned long long)(rb.y - rb.x);
      } else {
        v1g_walk_rec<R_>(a, basis_s, lane, (int)(ent >> 24),
                         a.rec_rowptr + (int64_t)(n0 + (int)(ent & 0xffffff)) * D, t, c_rec_ev);
      }
    }
    if (tid == 0) c_spikes += (unsigned long long)nspk;
    // LGN events of step t+1.  Dependent loads are spread over iterations and handed over in shared
    // memory: thread 0 fetches the bounds of the events of step t+3, every warp fetches its first
    // event of step t+2 (bounds known since the previous iteration), and what is left for now is
    // event (prefetched, with the bounds of its synapse row) -> synapse records -> atomics.
    // (asynchronous copies straight into shared memory: no register holds a value in flight)
    if (tid == 0) {
      int* bd = &s_misc[8 + 2 * ((t + 3) & 3)];
      if (t + 3 < a.T) {
        const int64_t spt = (int64_t)a.B * a.lgn_nseg;
        cp_async_4(bd, a.lgn_off + (int64_t)(t + 3) * spt);
        cp_async_4(bd + 1, a.lgn_off + (int64_t)(t + 4) * spt);
      } else {
        bd[0] = bd[1] = 0;
      }
    }
    if (lane == 0) {
      uint4* dst = &lgn_ent_s[(t & 1) * NW + warp];  // read in the next iteration (step t+2)
      const int e = s_misc[8 + 2 * ((t + 2) & 3)] + gw;
      if (t + 2 < a.T && e < s_misc[9 + 2 * ((t + 2) & 3)])
        cp_async_16(dst, a.lgn_ent4 + e);
      else
        *dst = make_uint4(0u, 0u, 0u, 0u);
    }
    if (t + 1 < a.T) {
      const int slot1 = (t + 1) % K;
      const int e0 = s_misc[8 + 2 * ((t + 1) & 3)], e1 = s_misc[9 + 2 * ((t + 1) & 3)];
      if (lgn8) {
        uint4 ent = lgn_ent_s[((t + 1) & 1) * NW + warp];
        ent.x = __shfl_sync(0xffffffffu, ent.x, 0);
        ent.y = __shfl_sync(0xffffffffu, ent.y, 0);
        ent.z = __shfl_sync(0xffffffffu, ent.z, 0);
        for (int e = e0 + gw; e < e1; e += gnw) {
          if (e != e0 + gw) ent = a.lgn_ent4[e];  // more events than warps in the grid
          v1g_scatter_row8<R_>(a, a.lgn_syn8, basis_s, lane, (int)(ent.x >> 24), (int)ent.y, (int)ent.z, slot1, false);
          if (lane == 0) {
            c_lgn_rows += 1;
            c_lgn_ev += (unsigned long long)(ent.z - ent.y);
          }
        }
      } else {
        v1g_scatter_lgn<R_>(a, basis_s, lane, gw, gnw, e0, e1, slot1, c_lgn_rows, c_lgn_ev);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // own copies landed; the barrier at the top of the next iteration publishes them
    if (prof) {
      const unsigned long long ph3 = gtime();
      ph_barrier += ph1 - ph0;
      ph_dense += ph2 - ph1;
      ph_scatter += ph3 - ph2;
    }
  }
  // ---- full barrier, then bring psc / psc_rise up to step T-1 ----
  __syncthreads();
  if (ctl) {
    if (ok && a.T >= 1) v1g_arrive(v1g_phase_counter(a.barrier, a.T));
    const unsigned long long target = v1g_phase_target(a.T, G);
    if (ok) {
      if (v1g_wait(v1g_phase_counter(a.barrier, a.T), target, a.spin_limit, a.status) < target) s_misc[1] = 1;
    }
  }
  __syncthreads();
  ok = ok && !s_misc[1];
  if (ok && a.T >= 1) {
    for (int s = max(a.T - 2, 0); s < a.T; ++s) {
      __syncthreads();
      for (int i = tid; i < nb; i += NT) {
        const int b = i / a.n_bkg, j = i - b * a.n_bkg;
        s_cnt[j * BP + b] = a.bkg_counts[((int64_t)b * a.T + s) * a.n_bkg + j];
      }
      __syncthreads();
      if (active) {
        float* rp = a.ring + ((int64_t)(s % K) * B_ * R_) * Np + n;
#pragma unroll
        for (int b = 0; b < B_; ++b) {
          float Gs[R_];
          bkg_gather(W1{}, b, s_cnt, Gs);
#pragma unroll
          for (int r = 0; r < R_; ++r) {
            const float in = __ldcg(rp + (int64_t)(b * R_ + r) * Np);
            __stcg(rp + (int64_t)(b * R_ + r) * Np, 0.f);
            const float prv = PR(b, r);
            if (s == a.T - 1) PSC(b, r) = PSC(b, r) * a.sd[r] + a.dtsd[r] * prv;
            PR(b, r) = prv * a.sd[r] + ((in + Gs[r]) * a.lr_scale) * a.pinit[r];
          }
        }
      }
    }
  }
  if (prof) {
    unsigned long long* o = a.phase_ns + 4 * blockIdx.x;
    o[0] = ph_dense;
    o[1] = ph_scatter;
    o[2] = ph_barrier;
    o[3] = gtime() - ph[3];
  }
  if (have_state && ok && active) {
#pragma unroll
    for (int b = 0; b < B_; ++b) {
      const int64_t g = (int64_t)b * N + n;
      a.st.v[g] = v[b];
      a.st.r[g] = (int8_t)(rh[b] >> 8);
      a.st.asc[2 * g] = *as_row(b, 0);
      a.st.asc[2 * g + 1] = *as_row(b, 1);
#pragma unroll
      for (int r = 0; r < R_; ++r) {
        a.st.psc[g * R_ + r] = PSC(b, r);
        a.st.psc_rise[g * R_ + r] = PR(b, r);
      }
      for (int d = 0; d < D; ++d) a.st.z_buf[((int64_t)b * D + d) * N + n] = (rh[b] >> d) & 1u ? 1.f : 0.f;
    }
  }
  if (lane == 0) {
    V1GCounters* c = (V1GCounters*)a.counters;
    if (c_rec_ev) atomicAdd(&c->rec_events, c_rec_ev);
    if (c_lgn_rows) atomicAdd(&c->lgn_rows, c_lgn_rows);
    if (c_lgn_ev) atomicAdd(&c->lgn_events, c_lgn_ev);
    if (tid == 0 && c_spikes) {
      atomicAdd(&c->spikes, c_spikes);
      atomicAdd(&c->rec_rows, c_spikes * (unsigned long long)D);
    }
  }
}

// Background rows and events of a rollout: every synapse of a node with a count is delivered once, whatever
// the block.  Counted here and not where they are delivered: there it took 4 of 26 instructions per
// synapse and pair of rows.
__global__ void __launch_bounds__(256) count_bkg_kernel(const int32_t* __restrict__ counts, int64_t total, int n_bkg,
                                                        const int32_t* __restrict__ rowptr,
                                                        unsigned long long* __restrict__ counters) {
  unsigned long long rows = 0, events = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    if (counts[i] > 0) {
      const int j = (int)(i % n_bkg);
      rows += 1;
      events += (unsigned long long)(rowptr[j + 1] - rowptr[j]);
    }
  rows = v1g_warp_sum(rows);
  events = v1g_warp_sum(events);
  if ((threadIdx.x & 31) == 0 && rows) {
    V1GCounters* c = (V1GCounters*)counters;
    atomicAdd(&c->bkg_rows, rows);
    atomicAdd(&c->bkg_events, events);
  }
}

template <int R_, int B_>
int launch(V1GHandle* h, const FwdArgs& a, int grid, size_t smem, cudaStream_t st) {
  auto kern = rollout_fwd_reg_kernel<R_, B_>;
  V1G_CUDA(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  V1G_CUDA(h, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem));
  if (per_sm < 1 || grid > per_sm * h->n_sms)
    return v1g_fail(h, V1G_ERANGE, "rollout grid of %d blocks cannot be co-resident (%d per SM)", grid, per_sm);
  void* args[] = {(void*)&a};
  V1G_CUDA(h, cudaEventRecord(h->ev[0], st));
  V1G_CUDA(h, cudaLaunchCooperativeKernel((void*)kern, dim3(grid), dim3(NT), args, smem, st));
  V1G_CUDA(h, cudaEventRecord(h->ev[1], st));
  h->ev_valid[0] = true;
  const int64_t n_counts = (int64_t)a.B * a.T * a.n_bkg;
  count_bkg_kernel<<<(unsigned)std::min<int64_t>((n_counts + 1023) / 1024, h->n_sms), 256, 0, st>>>(
      a.bkg_counts, n_counts, a.n_bkg, a.bkg_rowptr, a.counters);
  V1G_CUDA(h, cudaGetLastError());
  v1g_count_launches(2);
  return V1G_OK;
}

template <int R_>
int launch_b(V1GHandle* h, const FwdArgs& a, int grid, size_t smem, cudaStream_t st) {
  switch (a.B) {
    case 1: return launch<R_, 1>(h, a, grid, smem, st);
    case 2: return launch<R_, 2>(h, a, grid, smem, st);
    case 3: return launch<R_, 3>(h, a, grid, smem, st);
    case 4: return launch<R_, 4>(h, a, grid, smem, st);
    case 5: return launch<R_, 5>(h, a, grid, smem, st);
    case 6: return launch<R_, 6>(h, a, grid, smem, st);
    case 7: return launch<R_, 7>(h, a, grid, smem, st);
    case 8: return launch<R_, 8>(h, a, grid, smem, st);
    default: return V1G_ERANGE;
  }
}

}  // namespace

size_t v1g_fwd_reg_smem(const V1GHandle* h, int B, int chunkP, int bkg_cap) {
  auto al = [](size_t b) { return (b + 15) & ~(size_t)15; };
  const V1GConfig& c = h->cfg;
  return al(sizeof(float) * c.n_syn_types * c.n_receptors) + al(sizeof(uint32_t) * B * NT) +
         al(sizeof(float) * 2 * c.n_syn_types * ((c.n_receptors + 1) & ~1)) + al(sizeof(int) * 2 * ((B + 1) & ~1) * c.n_bkg) + al(sizeof(int) * 16) + al(sizeof(unsigned long long) * (4 * NW + 4)) + al(sizeof(int2) * NT) + al(sizeof(uint4) * 2 * NW) +
         al(sizeof(uint2) * bkg_cap) +
         al(sizeof(float) * B * c.n_receptors * NT) * (psc_in_smem(B) ? 2 : 1) +
         (asc_in_smem(B) ? al(sizeof(float) * B * 2 * NT) : 0);
}

int v1g_launch_fwd_reg(V1GHandle* h, const FwdArgs& a, int R, int grid, size_t smem,
                       cudaStream_t st) {
  if (R == 4) return launch_b<4>(h, a, grid, smem, st);
  if (R == 5) return launch_b<5>(h, a, grid, smem, st);
  return V1G_ERANGE;
}
