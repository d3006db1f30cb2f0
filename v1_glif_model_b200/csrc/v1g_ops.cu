// Operator-level kernels: one launch group per TensorFlow-level callable of the reference cell.
// These are the functional (state in -> state out) forms used for per-step parity and by the
// TensorFlow op shim; the throughput path is the fused rollout.
#include <algorithm>

#include "v1g_internal.h"

namespace {

struct DenseConsts {
  float sd[V1G_MAX_RECEPTORS], pinit[V1G_MAX_RECEPTORS], dtsd[V1G_MAX_RECEPTORS];
  float vd_keep, vd_drop, damp, width, gauss_std;
  int N, R, D, hard_reset, gauss;
};

// ------------------------------------------------------------------------------------------
// spike -> current scatter and weight gradient over the active columns (models.py:134-169, 833-857,
// 896-934 and 226-240)
// ------------------------------------------------------------------------------------------
// A warp looks at `group` neighbouring columns of one batch row, and for every positive entry walks the
// column's synapses; the positions never have to be listed, since nothing depends on their order (the
// three launches of an ordered compaction, per source and call, were a sixth of the time of a step of
// 5,000 neurons: 192 -> 162 us).  Sources
// with few columns and long rows (background) are spread by taking one column per warp and every
// `parts`-th pass of 32 synapses of its row.
struct ActiveSplit {
  int group, parts;
  int64_t groups_per_row, items;
};

template <typename F>
__device__ __forceinline__ void for_active(const ActiveSplit sp, const float* __restrict__ x, int64_t n_cols, int D, int n_src,
                                           const int32_t* __restrict__ rowptr, F&& walk) {
  const int lane = threadIdx.x & 31;
  const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t item = gw; item < sp.items; item += nw) {
    const int part = (int)(item % sp.parts);
    const int64_t g = item / sp.parts, b = g / sp.groups_per_row, c0 = (g - b * sp.groups_per_row) * sp.group;
    const int64_t col = c0 + lane;
    float xv = 0.f;
    if (lane < sp.group && col < n_cols) xv = x[b * n_cols + col];
    unsigned act = __ballot_sync(0xffffffffu, xv > 0.f);
    int j0 = 0, j1 = 0;
    if (xv > 0.f) {
      const int64_t row = (D > 1) ? (col % n_src) * D + col / n_src : col;
      j0 = rowptr[row];
      j1 = rowptr[row + 1];
    }
    while (act) {
      const int src = __ffs(act) - 1;
      act &= act - 1;
      const float mult = __shfl_sync(0xffffffffu, xv, src);
      const int first = __shfl_sync(0xffffffffu, j0, src), end = __shfl_sync(0xffffffffu, j1, src);
      walk(b, mult, first + 32 * part + lane, end, 32 * sp.parts);
    }
  }
}

__global__ void __launch_bounds__(256) scatter_fwd_kernel(
    const ActiveSplit sp, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ post,
    const float* __restrict__ w, const uint8_t* __restrict__ sid, const float* __restrict__ basis,
    const float* __restrict__ x, int64_t n_cols, int N, int R, int S, int D, int n_src, int is_bkg,
    float* __restrict__ i_flat) {
  extern __shared__ float basis_s[];
  for (int i = threadIdx.x; i < S * R; i += blockDim.x) basis_s[i] = basis[i];
  __syncthreads();
  for_active(sp, x, n_cols, D, n_src, rowptr, [&](int64_t b, float mult, int first, int end, int step) {
    for (int j = first; j < end; j += step) {
      float wv = w[j];
      if (is_bkg) wv = wv * mult;  // (w * n_pre_spikes) * basis, models.py:931
      const float* bs = basis_s + (int)sid[j] * R;
      float* dst = i_flat + (b * N + post[j]) * R;
      for (int r = 0; r < R; ++r) {
        const float c = wv * bs[r];
        if (c != 0.f) atomicAdd(dst + r, c);
      }
    }
  });
}

// d_w[syn] += sum_r dy[b,post,r]*basis[sid,r] for the synapses of active columns
// (models.py:226-240); the background source carries the Poisson count (autodiff of :931).
__global__ void __launch_bounds__(256) scatter_dw_kernel(
    const ActiveSplit sp, const int32_t* __restrict__ rowptr, const int32_t* __restrict__ post,
    const uint8_t* __restrict__ sid, const int32_t* __restrict__ perm,
    const float* __restrict__ basis, const float* __restrict__ x, const float* __restrict__ dy,
    int64_t n_cols, int N, int R, int S, int D, int n_src, int is_bkg, float* __restrict__ d_w) {
  extern __shared__ float basis_s[];
  for (int i = threadIdx.x; i < S * R; i += blockDim.x) basis_s[i] = basis[i];
  __syncthreads();
  for_active(sp, x, n_cols, D, n_src, rowptr, [&](int64_t b, float mult, int first, int end, int step) {
    for (int j = first; j < end; j += step) {
      const float* bs = basis_s + (int)sid[j] * R;
      const float* g = dy + (b * N + post[j]) * R;
      float s = 0.f;
      for (int r = 0; r < R; ++r) s += g[r] * bs[r];
      if (is_bkg) s = s * mult;
      atomicAdd(d_w + perm[j], s);
    }
  });
}

// ------------------------------------------------------------------------------------------
// d_x[b, col] = sum over the synapses of column col of w * sum_r basis[sid,r]*dy[b,post,r]
// (models.py:187-202; every synapse, active or not)
// ------------------------------------------------------------------------------------------
// Every synapse is read once for up to BP batch rows together.  What bounds the gather is one L2 sector
// per synapse: dy is laid out anew so that the values one synapse needs are neighbours, padded to BP in
// {1, 2, 4, 8} floats (32 bytes at most).  With few synapse types (PROJ) the basis is applied there too
// and a synapse reads one such row, its type's; otherwise it reads the R rows of its target.  Currents and
// both gradients of one step at 66,634 neurons, batch 5 (8 M synapses): 536 us with a pass over the
// synapses per batch row, 145 us with this.
constexpr int PROJ_MAX_TYPES = 8;

template <int BP, bool PROJ>
__global__ void __launch_bounds__(256) gather_rows_kernel(const float* __restrict__ dy, const float* __restrict__ basis,
                                                          int b0, int nb, int N, int R, int S, float* __restrict__ rows) {
  const int M = PROJ ? S : R;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < (int64_t)N * M; i += (int64_t)gridDim.x * blockDim.x) {
    const int n = (int)(i / M), m = (int)(i - (int64_t)n * M);
    float v[BP];
#pragma unroll
    for (int b = 0; b < BP; ++b) {
      v[b] = 0.f;
      if (b >= nb) continue;
      const float* g = dy + ((int64_t)(b0 + b) * N + n) * R;
      if (PROJ) {
        for (int r = 0; r < R; ++r) v[b] += g[r] * basis[m * R + r];
      } else {
        v[b] = g[m];
      }
    }
#pragma unroll
    for (int b = 0; b < BP; ++b) rows[i * BP + b] = v[b];
  }
}

template <int BP>
struct alignas(BP * 4) GatherRow {
  float v[BP];
};
// a whole row in one load: with 32 bytes as two loads every lane pays its own L1 line access twice
template <int BP>
__device__ __forceinline__ GatherRow<BP> load_row(const GatherRow<BP>* p) {
  if constexpr (BP == 8) {
    GatherRow<8> g;
    asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(g.v[0]), "=f"(g.v[1]), "=f"(g.v[2]), "=f"(g.v[3]), "=f"(g.v[4]), "=f"(g.v[5]), "=f"(g.v[6]), "=f"(g.v[7])
                 : "l"(p));
    return g;
  } else {
    return *p;
  }
}

// LPR lanes walk one row of the CSR, U synapses each at a time with all their loads in flight
template <int BP, bool PROJ, int LPR>
__global__ void __launch_bounds__(256) gather_dx_kernel(
    const int32_t* __restrict__ rowptr, const int32_t* __restrict__ post, const float* __restrict__ w,
    const uint8_t* __restrict__ sid, const float* __restrict__ basis, const float* __restrict__ rows, int64_t n_cols, int b0,
    int nb, int R, int S, int D, int n_src, float* __restrict__ d_x) {
  constexpr int U = 4;
  extern __shared__ float basis_s[];
  if (!PROJ) {
    for (int i = threadIdx.x; i < S * R; i += blockDim.x) basis_s[i] = basis[i];
    __syncthreads();
  }
  const GatherRow<BP>* rw = reinterpret_cast<const GatherRow<BP>*>(rows);
  const int l = threadIdx.x & (LPR - 1);
  const int64_t g0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LPR;
  const int64_t ng = ((int64_t)gridDim.x * blockDim.x) / LPR;
  // whole warps stay in the loop, so that the shuffles below always have all their lanes
  const int64_t n_it = (n_cols + ng - 1) / ng;
  int64_t row = g0;
  for (int64_t it = 0; it < n_it; ++it, row += ng) {
    const bool in = row < n_cols;
    const int j0 = in ? rowptr[row] : 0, j1 = in ? rowptr[row + 1] : 0;
    float acc[BP];
#pragma unroll
    for (int b = 0; b < BP; ++b) acc[b] = 0.f;
    for (int jb = j0 + l; jb < j1; jb += LPR * U) {
      int p[U], s[U];
      float wv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int j = jb + q * LPR;
        const bool ok = j < j1;
        p[q] = ok ? post[j] : 0;
        s[q] = ok ? (int)sid[j] : -1;
        wv[q] = ok ? w[j] : 0.f;
      }
      if (PROJ) {
        GatherRow<BP> gr[U];
#pragma unroll
        for (int q = 0; q < U; ++q)
          if (s[q] >= 0) gr[q] = load_row<BP>(rw + (int64_t)p[q] * S + s[q]);
#pragma unroll
        for (int q = 0; q < U; ++q)
          if (s[q] >= 0) {
#pragma unroll
            for (int b = 0; b < BP; ++b) acc[b] += wv[q] * gr[q].v[b];
          }
      } else {
#pragma unroll
        for (int q = 0; q < U; ++q) {
          if (s[q] < 0) continue;
          for (int r = 0; r < R; ++r) {
            const float wb = wv[q] * basis_s[s[q] * R + r];
            const GatherRow<BP> gr = load_row<BP>(rw + (int64_t)p[q] * R + r);
#pragma unroll
            for (int b = 0; b < BP; ++b) acc[b] += gr.v[b] * wb;
          }
        }
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1)
#pragma unroll
      for (int b = 0; b < BP; ++b) acc[b] += __shfl_xor_sync(0xffffffffu, acc[b], o);
    if (!in) continue;
    const int64_t col = (D > 1) ? (row % D) * n_src + row / D : row;
#pragma unroll
    for (int b = 0; b < BP; ++b)
      if (l == b && b < nb) d_x[(int64_t)(b0 + b) * n_cols + col] = acc[b];
  }
}

// ------------------------------------------------------------------------------------------
// dense update (models.py:979-1028) + spike, refractory gate and buffer shift (:1105-1117)
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) step_fwd_kernel(
    DenseConsts k, int B, const float* __restrict__ decay, const float* __restrict__ cf,
    const float* __restrict__ asc_decay, const float* __restrict__ asc_amps,
    const int32_t* __restrict__ tref, V1GState in, const float* __restrict__ rec_inputs,
    V1GState out, float* __restrict__ z_out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int N = k.N, R = k.R, D = k.D;
  if (i >= (int64_t)B * N) return;
  const int b = (int)(i / N), n = (int)(i - (int64_t)b * N);
  const float* zb = in.z_buf + (int64_t)b * D * N;
  const float prev_z = zb[n];
  float csum = 0.f;
  const int64_t o = i * R;
  for (int r = 0; r < R; ++r) {
    const float I = rec_inputs[o + r], pr = in.psc_rise[o + r], p = in.psc[o + r];
    out.psc_rise[o + r] = pr * k.sd[r] + I * k.pinit[r];
    out.psc[o + r] = p * k.sd[r] + k.dtsd[r] * pr;
    csum = (r == 0) ? p : csum + p;
  }
  const float a0 = in.asc[i * 2], a1 = in.asc[i * 2 + 1];
  out.asc[i * 2] = asc_decay[n * 2] * a0 + prev_z * asc_amps[n * 2];
  out.asc[i * 2 + 1] = asc_decay[n * 2 + 1] * a1 + prev_z * asc_amps[n * 2 + 1];
  const float c1 = csum + (a0 + a1);
  const float v = in.v[i];
  const float dv = v * k.vd_keep + v * k.vd_drop;
  float nv = (decay[n] * dv + cf[n] * c1) - prev_z;
  int nr = (int)in.r[i] + (int)prev_z * tref[n] - 1;
  nr = nr > 0 ? nr : 0;
  if (k.hard_reset && nr > 0) nv = 0.f;
  float z = ((nv - 1.f) > 0.f) ? 1.f : 0.f;
  if (nr > 0) z = 0.f;
  out.v[i] = nv;
  out.r[i] = (int8_t)nr;
  float* zo = out.z_buf + (int64_t)b * D * N;
  zo[n] = z;
  for (int d = 1; d < D; ++d) zo[(int64_t)d * N + n] = zb[(int64_t)(d - 1) * N + n];
  if (z_out) z_out[i] = z;
}

__device__ __forceinline__ float pseudo_h(float vs, const DenseConsts& k) {
  if (k.gauss) return expf(-(vs * vs) / (k.gauss_std * k.gauss_std)) * k.damp;
  float a = fabsf(vs);
  if (k.width != 1.f) a = a / k.width;
  return k.damp * fmaxf(1.f - a, 0.f);
}

__global__ void __launch_bounds__(256) step_bwd_kernel(
    DenseConsts k, int B, const float* __restrict__ decay, const float* __restrict__ cf,
    const float* __restrict__ asc_decay, V1GState g_out, const float* __restrict__ g_z,
    const float* __restrict__ g_v_out, const float* __restrict__ new_v,
    const int8_t* __restrict__ new_r, V1GState g_in, float* __restrict__ g_rec_inputs) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int N = k.N, R = k.R, D = k.D;
  if (i >= (int64_t)B * N) return;
  const int b = (int)(i / N), n = (int)(i - (int64_t)b * N);
  const float* gzb = g_out.z_buf ? g_out.z_buf + (int64_t)b * D * N : nullptr;
  float gz = g_z ? g_z[i] : 0.f;
  if (gzb) gz += gzb[n];
  const bool free_ = new_r[i] == 0;
  float gnv = (g_out.v ? g_out.v[i] : 0.f) + (g_v_out ? g_v_out[i] : 0.f);
  if (free_) gnv += gz * pseudo_h(new_v[i] - 1.f, k);
  if (k.hard_reset && !free_) gnv = 0.f;
  g_in.v[i] = decay[n] * k.vd_keep * gnv;
  const float gc1 = cf[n] * gnv;
  const int64_t o = i * R;
  for (int r = 0; r < R; ++r) {
    const float gpr = g_out.psc_rise ? g_out.psc_rise[o + r] : 0.f;
    const float gp = g_out.psc ? g_out.psc[o + r] : 0.f;
    g_in.psc[o + r] = k.sd[r] * gp + gc1;
    g_in.psc_rise[o + r] = k.sd[r] * gpr + k.dtsd[r] * gp;
    g_rec_inputs[o + r] = k.pinit[r] * gpr;
  }
  for (int q = 0; q < 2; ++q) {
    const float ga = g_out.asc ? g_out.asc[i * 2 + q] : 0.f;
    g_in.asc[i * 2 + q] = asc_decay[n * 2 + q] * ga + gc1;
  }
  if (g_in.z_buf) {
    float* go = g_in.z_buf + (int64_t)b * D * N;
    for (int d = 0; d < D - 1; ++d) go[(int64_t)d * N + n] = gzb ? gzb[(int64_t)(d + 1) * N + n] : 0.f;
    go[(int64_t)(D - 1) * N + n] = 0.f;
  }
}

DenseConsts make_consts(const V1GHandle* h) {
  DenseConsts k;
  const V1GConfig& c = h->cfg;
  for (int r = 0; r < V1G_MAX_RECEPTORS; ++r) {
    k.sd[r] = r < c.n_receptors ? h->syn_decay[r] : 0.f;
    k.pinit[r] = r < c.n_receptors ? h->psc_initial[r] : 0.f;
    k.dtsd[r] = c.dt * k.sd[r];
  }
  k.vd_keep = h->vd_keep;
  k.vd_drop = h->vd_drop;
  k.damp = c.dampening_factor;
  k.width = c.pseudo_width;
  k.gauss_std = c.gauss_std;
  k.N = c.n_neurons;
  k.R = c.n_receptors;
  k.D = c.max_delay;
  k.hard_reset = (c.flags & V1G_FLAG_HARD_RESET) ? 1 : 0;
  k.gauss = (c.flags & V1G_FLAG_PSEUDO_GAUSS) ? 1 : 0;
  return k;
}

int check_source(V1GHandle* h, int source, int batch) {
  if (source < 0 || source >= V1G_NSRC) return v1g_fail(h, V1G_EINVAL, "unknown source %d", source);
  if (!h->src[source].rowptr) return v1g_fail(h, V1G_ESTATE, "connectivity of source %d not set", source);
  if (!h->params_set) return v1g_fail(h, V1G_ESTATE, "neuron parameters not set");
  if (batch <= 0) return v1g_fail(h, V1G_EINVAL, "batch must be > 0");
  return V1G_OK;
}

ActiveSplit split_active(const V1GHandle* h, const V1GSource& s, int batch) {
  // about 32 warps per SM, each on as many columns as that leaves it (32 at most), and passes of 256
  // synapses where a row is longer than that
  const int64_t cols = (int64_t)batch * s.n_cols, warps = (int64_t)h->n_sms * 32;
  ActiveSplit sp;
  sp.group = 1;
  while (sp.group < 32 && cols / sp.group > warps) sp.group *= 2;
  const int64_t mean = s.n_cols > 0 ? s.nnz / s.n_cols : 0;
  sp.parts = (int)std::min<int64_t>(std::max<int64_t>(mean / 256, 1), 64);
  sp.groups_per_row = (s.n_cols + sp.group - 1) / sp.group;
  sp.items = sp.groups_per_row * batch * sp.parts;
  return sp;
}

unsigned active_blocks(const V1GHandle* h, const ActiveSplit& sp) {
  return (unsigned)std::max<int64_t>(std::min<int64_t>((sp.items + 7) / 8, (int64_t)h->n_sms * 8), 1);
}

template <int BP, bool PROJ>
int gather_dx(V1GHandle* h, const V1GSource& s, const float* dy, int b0, int nb, float* d_x, cudaStream_t st) {
  const int N = h->cfg.n_neurons, R = h->cfg.n_receptors, S = h->cfg.n_syn_types;
  const int64_t elems = (int64_t)N * (PROJ ? S : R);
  int rc;
  if ((rc = v1g_reserve(h, &h->gather_rows, &h->gather_rows_cap, elems * BP))) return rc;
  gather_rows_kernel<BP, PROJ><<<(unsigned)std::min<int64_t>((elems + 255) / 256, (int64_t)h->n_sms * 8), 256, 0, st>>>(
      dy, h->basis, b0, nb, N, R, S, h->gather_rows);
  const size_t smem = PROJ ? 0 : (size_t)S * R * sizeof(float);
  // rows of the recurrent source are short (one delay of one neuron): 8 lanes walk one, four rows per warp
  const int lpr = s.nnz / std::max<int64_t>(s.n_cols, 1) < 48 ? 8 : 32;
  const unsigned blocks = (unsigned)std::min<int64_t>((s.n_cols * lpr + 255) / 256, (int64_t)h->n_sms * 32);
  auto kern = lpr == 8 ? gather_dx_kernel<BP, PROJ, 8> : gather_dx_kernel<BP, PROJ, 32>;
  kern<<<blocks, 256, smem, st>>>(s.rowptr, s.post, s.w, s.sid, h->basis, h->gather_rows, s.n_cols, b0, nb, R, S, s.delays,
                                  s.n_src, d_x);
  v1g_count_launches(2);
  V1G_CUDA(h, cudaGetLastError());
  return V1G_OK;
}

}  // namespace

extern "C" int v1g_syn_currents_fwd(V1GHandle* h, int source, const float* x, int32_t batch,
                                    float* i_flat, void* stream) {
  if (!h) return V1G_EINVAL;
  int rc = check_source(h, source, batch);
  if (rc) return rc;
  if (!x || !i_flat) return v1g_fail(h, V1G_EINVAL, "v1g_syn_currents_fwd: null argument");
  cudaStream_t st = (cudaStream_t)stream;
  const V1GSource& s = h->src[source];
  const int N = h->cfg.n_neurons, R = h->cfg.n_receptors, S = h->cfg.n_syn_types;
  V1G_CUDA(h, cudaMemsetAsync(i_flat, 0, (size_t)batch * N * R * sizeof(float), st));
  if (s.nnz == 0) return V1G_OK;
  const ActiveSplit sp = split_active(h, s, batch);
  scatter_fwd_kernel<<<active_blocks(h, sp), 256, S * R * sizeof(float), st>>>(
      sp, s.rowptr, s.post, s.w, s.sid, h->basis, x, s.n_cols, N, R, S, s.delays, s.n_src,
      source == V1G_SRC_BKG, i_flat);
  v1g_count_launches(1);
  V1G_CUDA(h, cudaGetLastError());
  return V1G_OK;
}

extern "C" int v1g_syn_currents_bwd(V1GHandle* h, int source, const float* x, const float* dy,
                                    int32_t batch, float* d_x, float* d_w, void* stream) {
  if (!h) return V1G_EINVAL;
  int rc = check_source(h, source, batch);
  if (rc) return rc;
  if (!x || !dy) return v1g_fail(h, V1G_EINVAL, "v1g_syn_currents_bwd: null argument");
  cudaStream_t st = (cudaStream_t)stream;
  const V1GSource& s = h->src[source];
  const int N = h->cfg.n_neurons, R = h->cfg.n_receptors, S = h->cfg.n_syn_types;
  if (d_x && s.n_cols > 0) {
    const bool proj = S <= PROJ_MAX_TYPES;
    for (int b0 = 0; b0 < batch; b0 += 8) {
      const int nb = std::min(batch - b0, 8);
      if (nb == 1) rc = proj ? gather_dx<1, true>(h, s, dy, b0, nb, d_x, st) : gather_dx<1, false>(h, s, dy, b0, nb, d_x, st);
      else if (nb == 2) rc = proj ? gather_dx<2, true>(h, s, dy, b0, nb, d_x, st) : gather_dx<2, false>(h, s, dy, b0, nb, d_x, st);
      else if (nb <= 4) rc = proj ? gather_dx<4, true>(h, s, dy, b0, nb, d_x, st) : gather_dx<4, false>(h, s, dy, b0, nb, d_x, st);
      else rc = proj ? gather_dx<8, true>(h, s, dy, b0, nb, d_x, st) : gather_dx<8, false>(h, s, dy, b0, nb, d_x, st);
      if (rc) return rc;
    }
  }
  if (d_w && s.nnz > 0) {
    V1G_CUDA(h, cudaMemsetAsync(d_w, 0, (size_t)s.nnz * sizeof(float), st));
    const ActiveSplit sp = split_active(h, s, batch);
    scatter_dw_kernel<<<active_blocks(h, sp), 256, S * R * sizeof(float), st>>>(
        sp, s.rowptr, s.post, s.sid, s.perm, h->basis, x, dy, s.n_cols, N, R, S, s.delays, s.n_src,
        source == V1G_SRC_BKG, d_w);
    v1g_count_launches(1);
    V1G_CUDA(h, cudaGetLastError());
  }
  return V1G_OK;
}

static bool state_complete(const V1GState* s) {
  return s && s->z_buf && s->v && s->r && s->asc && s->psc_rise && s->psc;
}

extern "C" int v1g_step_fwd(V1GHandle* h, int32_t batch, const V1GState* in,
                            const float* rec_inputs, V1GState* out, float* z_out, void* stream) {
  if (!h) return V1G_EINVAL;
  if (!h->params_set) return v1g_fail(h, V1G_ESTATE, "neuron parameters not set");
  if (batch <= 0 || !state_complete(in) || !state_complete(out) || !rec_inputs)
    return v1g_fail(h, V1G_EINVAL, "v1g_step_fwd: bad argument");
  const int64_t total = (int64_t)batch * h->cfg.n_neurons;
  step_fwd_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      make_consts(h), batch, h->decay, h->cf, h->asc_decay, h->asc_amps, h->tref, *in, rec_inputs,
      *out, z_out);
  v1g_count_launches(1);
  V1G_CUDA(h, cudaGetLastError());
  return V1G_OK;
}

extern "C" int v1g_step_bwd(V1GHandle* h, int32_t batch, const V1GState* g_out, const float* g_z,
                            const float* g_v_out, const float* new_v, const int8_t* new_r,
                            V1GState* g_in, float* g_rec_inputs, void* stream) {
  if (!h) return V1G_EINVAL;
  if (!h->params_set) return v1g_fail(h, V1G_ESTATE, "neuron parameters not set");
  if (batch <= 0 || !g_out || !g_in || !new_v || !new_r || !g_rec_inputs || !g_in->v ||
      !g_in->asc || !g_in->psc || !g_in->psc_rise)
    return v1g_fail(h, V1G_EINVAL, "v1g_step_bwd: bad argument");
  const int64_t total = (int64_t)batch * h->cfg.n_neurons;
  step_bwd_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      make_consts(h), batch, h->decay, h->cf, h->asc_decay, *g_out, g_z, g_v_out, new_v, new_r,
      *g_in, g_rec_inputs);
  v1g_count_launches(1);
  V1G_CUDA(h, cudaGetLastError());
  return V1G_OK;
}
