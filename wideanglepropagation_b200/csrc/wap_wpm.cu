// WPM adaptive-binning forward (propagation.py:215-256, :358-387).
//
// Launch sequence for N slices, all in place on the caller's exit buffer:
//   wpm_slices_kernel          reference deltas and record of every slice (one launch)
//   row pass  (load, FFT)      psi0 -> row spectrum
//   for s in 0..N-1:
//     wpm_node_col_kernel s    column FFT, per field (factor, column IFFT) -> fields
//     wpm_node_row_kernel s    per field row IFFT, blend -> wave after slice s,
//                              then its row FFT (input of slice s+1)
//   wpm_col_kernel (dp mode)   |fftshift(fft2(exit))|^2
// with the fields of a few interpolation nodes (wap_wpm_nodes.cuh), or, for grids
// that reach the evanescent edge, wpm_col_kernel / wpm_row_kernel with the fields
// of the K reference indices.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "wap_internal.h"
#include "wap_passes.cuh"
#include "wap_wpm_nodes.cuh"

namespace wap {

// WPM vacuum propagator exp(i dz sqrt_c(k0^2 - k_perp^2)) in float64 on the
// 'xy' meshgrid of propagation.py:224-228 (rows: ky = 2 pi fftfreq(ny, dy)),
// rounded once to complex64, plus the float32 tables (2 pi f)^2 per axis and
// q = k0^2 - k_perp^2.  q is rounded once: near the evanescent edge the difference
// of the rounded terms (k0^2 is some 1e5) was off by as much as q, which put 2e-5
// into the exit wave of a 64 x 67 grid with a mode there.
struct HvacArgs {
  int ny, nx;
  double dy, dx, dz, k0;
  float2* hvac;
  float2* hvac_lo;
  float* ky2;
  float* kx2;
  float* q;
};

__global__ void wpm_vacuum_kernel(const HvacArgs a) {
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)a.ny * a.nx) return;
  const int iy = (int)(idx / a.nx), ix = (int)(idx % a.nx);
  const double ky = 2.0 * M_PI * fftfreq_d(iy, a.ny, a.dy);
  const double kx = 2.0 * M_PI * fftfreq_d(ix, a.nx, a.dx);
  const double q = a.k0 * a.k0 - (kx * kx + ky * ky);
  double re, im;
  if (q >= 0.0) {
    sincos(a.dz * sqrt(q), &im, &re);
  } else {
    re = exp(-a.dz * sqrt(-q));
    im = 0.0;
  }
  const float rh = (float)re, ih = (float)im;
  a.q[idx] = (float)q;
  a.hvac[idx] = make_float2(rh, ih);
  a.hvac_lo[idx] = make_float2((float)(re - (double)rh), (float)(im - (double)ih));
  if (ix == 0) a.ky2[iy] = (float)(ky * ky);
  if (iy == 0) a.kx2[ix] = (float)(kx * kx);
}

// ----------------------------------------------------------------------------
// the slices' reference values and records
// ----------------------------------------------------------------------------
struct WpmSlicesArgs {
  const float* V;            // (draws, n_slices, ny, nx)
  float* refs;               // (draws, n_slices, K) delta reference values
  WpmSlice* rec;             // (draws, n_slices)
  int n_px, n_slices, K;
  int use_nodes;             // 0: no node records (grids that reach the evanescent edge, few bins)
  float ri_a, ri_inv_den;
  double power, k0, qmin, dz;
};

// Nodes needed for a range of half width ah whose largest |a| is amax, or 0 if
// none up to `most` meets the tolerance.  Interpolation at r Chebyshev nodes of
// [-1, 1] is off by at most max|f^(r)| / (2^(r-1) r!), f = exp(i g):
// |f^(r)| / r! <= [z^r] exp(T z + sum_{m>=2} b_m z^m), T bounding the slope of
// g (the variation of dz / (2 sqrt(q + a)) about kappa) and b_m the Taylor
// coefficients of the square root, 2 theta |binom(1/2, m)| y^(m-1) with
// theta = dz ah / (2 sqrt(q)) and y = ah / q at the smallest q.
__host__ __device__ inline int wpm_node_count(double ah, double amax, double qmin, double k0, double dz, int most) {
  const double qe = qmin - amax - ah;
  const double y = ah / qe, th = fabs(dz) * ah / (2.0 * sqrt(qe));
  double g[kWpmMaxNodes + 1], e[kWpmMaxNodes + 1];
  g[1] = fabs(dz) * ah * (1.0 / sqrt(qmin) - 1.0 / k0) / 4.0 + th * amax / (2.0 * qe);
  double b = 0.5, ym = 1.0;
  for (int m = 2; m <= kWpmMaxNodes; ++m) {
    b *= fabs(0.5 - (m - 1)) / m;
    ym *= y;
    g[m] = 2.0 * th * b * ym;
  }
  e[0] = 1.0;
  double half = 2.0;
  for (int r = 1; r <= kWpmMaxNodes; ++r) {
    double s = 0.0;
    for (int m = 1; m <= r; ++m) s += m * g[m] * e[r - m];
    e[r] = s / r;
    half *= 0.5;   // 2^-(r-1)
    if (e[r] * half <= kWpmNodeTol) return r <= most ? r : 0;
  }
  return 0;
}

// Per (slice, draw): min / max over the slice of n^2 - 1 = V (a + V) inv_den, in
// which delta = n - 1 grows (values without a real n are left out, as a NaN
// delta always was), the K reference values delta_min + (delta_max - delta_min) t_k^p in
// float64, and the slice's record.  One cluster of kWpmCluster CTAs per slice: each
// reduces its share with eight 16-byte loads in flight per thread, the first CTA
// folds the shares through distributed shared memory.  One CTA per slice (the
// loads of a whole slice in one SM) took 41 us at 512^2 for any slice count.
constexpr int kWpmCluster = 8;
constexpr int kWpmSliceThreads = 512;

static __global__ void __cluster_dims__(kWpmCluster, 1, 1) __launch_bounds__(kWpmSliceThreads)
wpm_slices_kernel(const WpmSlicesArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  constexpr int kInFlight = 8;
  const int s = blockIdx.x / kWpmCluster, d = blockIdx.y;
  const long long row = (long long)d * a.n_slices + s;
  const float* v = a.V + row * a.n_px;
  float lo = INFINITY, hi = -INFINITY;
  auto fold = [&](float volts) {
    const float r = volts * (a.ri_a + volts) * a.ri_inv_den;
    if (r >= -1.0f && r < INFINITY) {
      lo = fminf(lo, r);
      hi = fmaxf(hi, r);
    }
  };
  const int first = (int)cl.block_rank() * kWpmSliceThreads + threadIdx.x, step = kWpmCluster * kWpmSliceThreads;
  if ((a.n_px & 3) == 0 && (reinterpret_cast<uintptr_t>(a.V) & 15) == 0) {
    const float4* v4 = reinterpret_cast<const float4*>(v);
    const int n4 = a.n_px >> 2;
    int i = first;
    for (; i + (kInFlight - 1) * step < n4; i += kInFlight * step) {
      float4 q[kInFlight];
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) q[u] = __ldg(v4 + i + u * step);
#pragma unroll
      for (int u = 0; u < kInFlight; ++u) { fold(q[u].x); fold(q[u].y); fold(q[u].z); fold(q[u].w); }
    }
    for (; i < n4; i += step) {
      const float4 q = __ldg(v4 + i);
      fold(q.x); fold(q.y); fold(q.z); fold(q.w);
    }
  } else {
    for (int i = first; i < a.n_px; i += step) fold(__ldg(v + i));
  }
  __shared__ float slo[32], shi[32];
  __shared__ float part[2];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    slo[w] = lo;
    shi[w] = hi;
  }
  __syncthreads();
  if (w == 0) {
    constexpr int nw = kWpmSliceThreads / 32;
    lo = l < nw ? slo[l] : INFINITY;
    hi = l < nw ? shi[l] : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (l == 0) {
      part[0] = lo;
      part[1] = hi;
    }
  }
  cl.sync();
  if (cl.block_rank() == 0 && w < 2) {
    lo = INFINITY;
    hi = -INFINITY;
    if (l < kWpmCluster) {
      const float* p = cl.map_shared_rank(part, l);
      lo = p[0];
      hi = p[1];
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    lo = __shfl_sync(0xffffffffu, lo, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    const double dlo = wpm_delta(lo), dhi = wpm_delta(hi);
    if (w == 0) {
      float* out = a.refs + row * a.K;
      for (int k = l; k < a.K; k += 32) {
        // numpy linspace(0, 1, K): k * (1/(K-1)), last point exactly 1
        const double tk = (k == a.K - 1) ? 1.0 : (double)k * (1.0 / (double)(a.K - 1));
        const double tp = (a.power == 1.0) ? tk : pow(tk, a.power);
        out[k] = (float)(dlo + (dhi - dlo) * tp);
      }
    } else if (l == 0) {
      int nf = a.K, nodes = 0;
      float fxc = 0.f, finv = 0.f, fa0 = 0.f;
      const double k02 = a.k0 * a.k0;
      const double alo = k02 * dlo * (2.0 + dlo), ahi = k02 * dhi * (2.0 + dhi);
      const double ac = 0.5 * (alo + ahi), ah = 0.5 * (ahi - alo), amax = fmax(fabs(alo), fabs(ahi));
      // (a comparison with a NaN is false: such slices keep the K references)
      if (a.use_nodes && ah >= 0.0 && amax <= a.qmin * 0.125 && dlo > -0.5) {
        const int n = wpm_node_count(ah, amax, a.qmin, a.k0, a.dz, min(kWpmMaxNodes, a.K - 1));
        if (n > 0) {
          nf = n;
          nodes = 1;
          fxc = (float)(ac / k02);
          finv = ah > 0.0 ? (float)(k02 / ah) : 0.f;
          const int c = n >> 1;   // the node nearest the centre
          double tau[kWpmMaxNodes];
          for (int j = 0; j < n; ++j) {
            const int m = j == 0 ? c : (j <= c ? j - 1 : j);
            tau[j] = (2 * m + 1 == n) ? 0.0 : cos((2 * m + 1) * M_PI / (2.0 * n));
          }
          fa0 = (float)(ac + ah * tau[0]);
          for (int j = 0; j < n; ++j) {
            double p = 1.0;
            int i = 0;
            for (int m = 0; m < n; ++m) {
              if (m == j) continue;
              p *= tau[j] - tau[m];
              a.rec[row].other[j][i++] = (float)tau[m];
            }
            a.rec[row].da[j] = (float)(ah * (tau[j] - tau[0]));
            a.rec[row].bw[j] = (float)(1.0 / p);
          }
        }
      }
      WpmSlice& r = a.rec[row];
      r.nf = nf;
      r.nodes = nodes;
      r.xc = fxc;
      r.inv_xh = finv;
      r.a0 = fa0;
      r.dlo = (float)dlo;
      r.inv_range = dhi > dlo ? (float)(1.0 / (dhi - dlo)) : 0.f;
    }
  }
  cl.sync();   // the shares stay readable until the first CTA has them
}

// ----------------------------------------------------------------------------
// launches of the interpolating passes: eight elements per thread at every size
// ----------------------------------------------------------------------------
constexpr int kNodeE = 8;

template <class K>
static cudaError_t node_smem(K kern, size_t smem) {
  return beyond_default_smem(smem)
             ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
             : cudaSuccess;
}

// Whether a pass of `lines` lines of n points leaves the chip waiting on each
// warp's chain of transforms, so that a line's fields go to several groups: up to
// two one-group warps per scheduler.  Measured per call, K = 16, split / not (when the
// line was drawn): one 512^2 probe x 200 slices 3.53 / 4.41 ms, four 256^2 probes x 100 1.55 / 2.07 ms;
// two 512^2 probes x 60 2.01 / 1.67 ms, one 1024^2 probe x 40 3.62 / 3.02 ms.
static bool node_split(int n, long long lines) { return lines * (n / kNodeE) <= 148LL * 256; }

// Blocks that share the K fields of a tile where a slice has no nodes: as many as the
// chip holds beside the `ctas` of the pass (`per_sm` threads an SM), and at least two
// fields for every group of each.
static int node_shares(long long ctas, int threads, int per_sm, int K, int groups) {
  return (int)std::max(1LL, std::min<long long>(148LL * per_sm / threads / ctas, K / (2 * groups)));
}

// Whether slices of a call may lack nodes with enough bins to share out (wpm_node_count
// for an index whose square goes from 1 to 1 + kWpmIndexRange, 15 kV at 300 keV).  The
// blocks that would share return from slices with nodes, but hold up the next pass's
// early launch: 256^2, K = 128, 12.3 us a slice without them, 13.0 with.  Slices that
// have no nodes take 234 us without them, 100 with.
constexpr double kWpmIndexRange = 0.0625;
static bool node_sharing(int K, double k0, double qmin, double dz) {
  const double k02 = k0 * k0, amax = kWpmIndexRange * k02;
  return K >= 16 && !(amax <= 0.125 * qmin && wpm_node_count(0.5 * amax, amax, qmin, k0, dz, kWpmMaxNodes) > 0);
}

template <int N, int G>
static cudaError_t launch_node_col_t(const WpmNodeColArgs& a, int nb, cudaStream_t st) {
  constexpr int T = N / kNodeE;
  // columns per CTA: eight (64-byte row segments) within the thread limit, four
  // when eight would leave SMs without a CTA
  int w = 8;
  while (w > 1 && (w * T * G > node_col_threads(N, G) || w > a.c.nx)) w >>= 1;
  if (w == 8 && (long long)(a.c.nx / w) * nb < 148 && 4 * T >= 32) w = 4;
  const size_t smem = (size_t)N * w * G * sizeof(float2) + FFTPlan<N, kNodeE>::TW_SIZE * sizeof(float4);
  const long long ctas = (long long)(a.c.nx / w) * nb;
  const int per_sm = G > 1 || N >= 2048 ? 512 : 768;
  const int z = a.sharing ? node_shares(ctas, w * T * G, per_sm, a.c.K, G) : 1;
  auto kern = z > 1 ? wpm_node_col_kernel<N, kNodeE, G, true> : wpm_node_col_kernel<N, kNodeE, G, false>;
  cudaError_t e = node_smem(kern, smem);
  if (e != cudaSuccess) return e;
  count_launch();
  return launch_pdl(kern, dim3(a.c.nx / w, nb, z), w * T * G, smem, st, a);
}

template <int N, int G>
static cudaError_t launch_node_row_t(WpmNodeRowArgs a, int nb, cudaStream_t st) {
  constexpr int T = N / kNodeE;
  // rows per CTA: kRowThreads threads per group (or half that with several
  // groups), fewer while SMs would be left without two CTAs; whole warps
  int rows = std::max(1, (G > 1 ? kRowThreads / 2 : kRowThreads) / T);
  while (rows > 1 && (rows > a.r.ny || ((long long)(a.r.ny / rows) * nb < 296 && rows * T * G > 128 && rows * T > 32)))
    rows >>= 1;
  // twiddles, pixel blends (28 bytes each), the groups' exchange segments, references
  const size_t smem = FFTPlan<N, kNodeE>::TW_SIZE * sizeof(float4) + (size_t)rows * N * 28 +
                      (size_t)rows * G * RowCfg<N, kNodeE>::PADN * sizeof(float2) + (size_t)a.r.K * sizeof(float);
  const long long ctas = (long long)(a.r.ny / rows) * nb;
  int z = a.sharing ? node_shares(ctas, rows * G * T, G > 1 ? 1024 : 768, a.r.K - 1, G) : 1;
  a.r.kpg = (a.r.K - 2 + z) / z;
  z = (a.r.K - 2 + a.r.kpg) / a.r.kpg;
  auto kern = z > 1 ? wpm_node_row_kernel<N, kNodeE, G, true> : wpm_node_row_kernel<N, kNodeE, G, false>;
  cudaError_t e = node_smem(kern, smem);
  if (e != cudaSuccess) return e;
  count_launch();
  return launch_pdl(kern, dim3(a.r.ny / rows, nb, z), rows * G * T, smem, st, a);
}

#define WAP_NODE_SIZES(M) M(32) M(64) M(128) M(256) M(512) M(1024) M(2048)
#define WAP_NODE_COL(M)                                                                                   \
  case M:                                                                                                 \
    return node_split(M, (long long)a.c.nx * nb) ? launch_node_col_t<M, node_col_groups(M)>(a, nb, st)    \
                                                 : launch_node_col_t<M, 1>(a, nb, st);
#define WAP_NODE_ROW(M)                                                                                   \
  case M:                                                                                                 \
    return node_split(M, (long long)a.r.ny * nb) ? launch_node_row_t<M, node_row_groups(M)>(a, nb, st)    \
                                                 : launch_node_row_t<M, 1>(a, nb, st);
static cudaError_t launch_node_col(int n, const WpmNodeColArgs& a, int nb, cudaStream_t st) {
  switch (n) { WAP_NODE_SIZES(WAP_NODE_COL) default: return cudaErrorInvalidValue; }
}
static cudaError_t launch_node_row(int n, const WpmNodeRowArgs& a, int nb, cudaStream_t st) {
  switch (n) { WAP_NODE_SIZES(WAP_NODE_ROW) default: return cudaErrorInvalidValue; }
}

// twiddles and tile counts of the interpolating passes (plan creation)
int wpm_node_twiddles(wap_plan* p) {
  const size_t tiles = (size_t)p->ny * std::min(p->max_batch, 65535) * sizeof(unsigned);
  cudaError_t err = cudaMalloc(&p->wn_tiles, tiles);
  if (err == cudaSuccess) err = cudaMemset(p->wn_tiles, 0, tiles);
  if (err != cudaSuccess) return cuda_fail(err, "WPM tile counts");
  for (int which = 0; which < 2; ++which) {
    float4*& d = which == 0 ? p->wn_tw_row : p->wn_tw_col;
    const std::vector<float4> h = twiddle_table(which == 0 ? p->nx : p->ny, kNodeE);
    cudaError_t e = cudaMalloc(&d, h.size() * sizeof(float4));
    if (e == cudaSuccess) e = cudaMemcpy(d, h.data(), h.size() * sizeof(float4), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      cudaFree(d);
      d = nullptr;
      return cuda_fail(e, "WPM twiddles");
    }
  }
  return WAP_OK;
}

// largest (2 pi f)^2 of numpy.fft.fftfreq(n, d)
static double k2_max(int n, double d) {
  const double k = 2.0 * M_PI * (double)(n / 2) / ((double)n * d);
  return k * k;
}

// Reference values and records of every slice.  Interpolation needs a grid that
// stays clear of the evanescent edge (k0^2 above the largest k_perp^2).  Its passes
// also serve the slices that then find no node count below K, with their K reference
// fields: few bins, where they beat the split reference kernels (512^2, K = 4: 0.83
// against 1.84 ms for 40 slices), and strong slices (node_sharing).  Where those fill
// the chip they are the slower by up to a quarter (eight 256^2 probes, K = 32, 10
// slices: 2.01 against 1.63 ms); the grids that reach the edge keep the reference kernels.
static int wpm_slices(wap_plan* p, const float* V, int n_slices, int n_draws, const Physics& ph, double dz,
                      double sampling_y, double sampling_x, double power_spacing, WpmNodeScalars* out,
                      cudaStream_t st) {
  const int K = p->n_bins;
  const size_t rows = (size_t)n_draws * n_slices;
  cudaError_t e;
  if (rows * K > p->refs_cap) {
    drop_outgrown(p, p->refs, p->refs_captured);
    p->refs = nullptr;
    p->refs_cap = 0;
    if ((e = cudaMalloc(&p->refs, rows * K * sizeof(float))) != cudaSuccess) return cuda_fail(e, "cudaMalloc(refs)");
    p->refs_cap = rows * K;
  }
  if (rows > p->slices_cap) {   // (grows with refs: K is the plan's)
    drop_outgrown(p, p->slices, p->refs_captured);
    p->refs_captured = false;
    p->slices = nullptr;
    p->slices_cap = 0;
    if ((e = cudaMalloc(&p->slices, rows * sizeof(WpmSlice))) != cudaSuccess)
      return cuda_fail(e, "cudaMalloc(WPM records)");
    p->slices_cap = rows;
  }
  if (stream_capture(st) == 1) p->refs_captured = true;
  const double qmin = ph.k0 * ph.k0 - (k2_max(p->ny, sampling_y) + k2_max(p->nx, sampling_x));
  out->nodes = qmin > 0.0 && std::fabs(dz) >= 1e-6;
  if (out->nodes) {
    const double inv_root = 0.5 * (1.0 / std::sqrt(qmin) + 1.0 / ph.k0), qbar = 1.0 / (inv_root * inv_root);
    out->kappa = (float)(0.5 * dz * inv_root);
    const double kk = 0.5 * dz * inv_root * ph.k0 * ph.k0;
    out->kk = make_float2((float)kk, (float)(kk - (double)(float)kk));
    out->dq = (float)(qbar - ph.k0 * ph.k0);
    out->inv_qbar = (float)(1.0 / qbar);
    out->inv_root_qbar = (float)inv_root;
    out->sharing = node_sharing(K, ph.k0, qmin, dz);
  }
  const long long plane = (long long)p->ny * p->nx;
  const WpmSlicesArgs a{V, p->refs, p->slices, (int)plane, n_slices, K, out->nodes ? 1 : 0, (float)ph.ri_a,
                        (float)ph.ri_inv_den, power_spacing, ph.k0, qmin, dz};
  const ProfToken tok = prof_begin(WAP_KIND_WPM_BINS, st);
  count_launch();
  wpm_slices_kernel<<<dim3(n_slices * kWpmCluster, n_draws), kWpmSliceThreads, 0, st>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "wpm_slices_kernel");
  prof_end(tok, st, 4.0 * plane * n_slices * n_draws);
  return WAP_OK;
}

WpmNodeColArgs wpm_node_col_args(const wap_plan* p, const WpmColArgs& c, const WpmNodeScalars& nodes) {
  WpmNodeColArgs n{c,          p->slices,      nodes.kappa,         nodes.dq, nodes.inv_qbar, nodes.inv_root_qbar,
                   4.0f / (c.dz * c.dz), nodes.sharing};
  n.c.tw = p->wn_tw_col;
  return n;
}
WpmNodeRowArgs wpm_node_row_args(const wap_plan* p, const WpmRowArgs& w, const WpmNodeScalars& nodes, double power) {
  WpmNodeRowArgs n{w, p->slices, p->wn_tiles, nodes.kk, power == 1.0 ? 1 : power == 2.0 ? 2 : 0, nodes.sharing};
  n.r.tw = p->wn_tw_row;
  return n;
}

// Slices [0, n_slices) of nb probes from the fields of interpolation nodes.
static int node_slices(const wap_plan* p, const WpmNodeScalars& nodes, const WpmColArgs& c, const WpmRowArgs& w,
                       double power, int n_slices, int nb, float2* stack, cudaStream_t st) {
  const long long plane = (long long)p->ny * p->nx;
  WpmNodeColArgs nc = wpm_node_col_args(p, c, nodes);
  WpmNodeRowArgs nr = wpm_node_row_args(p, w, nodes, power);
  nr.r.blend = p->blend;
  cudaError_t e;
  for (int s = 0; s < n_slices; ++s) {
    nc.c.slice = nr.r.slice = s;
    ProfToken tok = prof_begin(WAP_KIND_WPM_COL, st);
    if ((e = launch_node_col(p->ny, nc, nb, st)) != cudaSuccess) return cuda_fail(e, "wpm column pass");
    // wave in, one field out at least, vacuum propagator once
    prof_end(tok, st, 16.0 * plane * nb + 8.0 * plane);
    nr.r.last = (s == n_slices - 1);
    nr.r.snap = stack ? stack + (long long)s * plane : nullptr;
    tok = prof_begin(WAP_KIND_WPM_ROW, st);
    if ((e = launch_node_row(p->nx, nr, nb, st)) != cudaSuccess) return cuda_fail(e, "wpm row pass");
    prof_end(tok, st, (20.0 + (nr.r.last ? 8.0 : 0.0) + (nr.r.snap ? 8.0 : 0.0)) * plane * nb);
  }
  return WAP_OK;
}

// The same from the fields of the K reference indices.
static int reference_slices(const wap_plan* p, const Physics& ph, const float* V, const int32_t* draw, WpmColArgs c,
                            WpmRowArgs w, int n_slices, int b0, int nb, float2* exit, float2* stack, cudaStream_t st) {
  const int K = p->n_bins;
  const long long plane = (long long)p->ny * p->nx;
  const int rows = rows_per_cta(p->nx, p->row_e, p->ny, 65535);   // the bin split below fills the chip
  cudaError_t e;
  // Few probes leave most SMs idle (a 512^2 probe is 128 column and 128 row
  // CTAs): then the K bins are split across CTA groups - each column CTA
  // redoes the column FFT for its share of the bins, each row CTA blends the
  // pixels whose left bin is in its share, and a row pass applies the row FFT.
  // The group count minimises (waves of resident CTAs) x (transforms per CTA).
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device);
  const int col_slots = std::max(1, wpm_col_occupancy(p->ny, p->col_e, p->col_w, K)) * sms;
  const int row_slots = std::max(1, wpm_row_occupancy(p->nx, p->row_e, rows, K)) * sms;
  // Bins per group (the launched group count is ceil(units / per)).  Column
  // CTA: 1 + per transforms; row CTA: K transforms unsplit, else per + 1 and
  // the row pass that follows (counted as one more).
  auto best_per = [&](long long ctas0, int slots, int units, bool col) {
    int best = units;
    double best_cost = 1e300;
    for (int per = units; per >= 1; --per) {
      const long long g = (units + per - 1) / per;
      const double waves = std::ceil((double)(ctas0 * g) / slots);
      const double work = col ? 1.0 + per : (g == 1 ? (double)K : per + 2.0);
      if (waves * work < best_cost) {
        best_cost = waves * work;
        best = per;
      }
    }
    return best;
  };

  c.kpg = best_per((long long)(p->nx / p->col_w) * nb, col_slots, K, true);
  w.kpg = best_per((long long)(p->ny / rows) * nb, row_slots, K - 1, false);
  const int gr = (K - 1 + w.kpg - 1) / w.kpg;
  w.blend = gr > 1 ? p->blend : nullptr;
  RowArgs fin = base_row_args(p, ph, V, n_slices, draw);   // the row FFT after a bin-split blend
  fin.src = p->blend;
  fin.src_bstride = plane;
  fin.shifts = nullptr;
  fin.flags = ROW_LOAD_SRC | ROW_FFT;
  for (int s = 0; s < n_slices; ++s) {
    c.slice = s;
    c.dp_mode = 0;
    ProfToken tok = prof_begin(WAP_KIND_WPM_COL, st);
    if ((e = launch_wpm_col(p->ny, p->col_e, c, nb, p->col_w, st)) != cudaSuccess) return cuda_fail(e, "wpm column pass");
    // wave in, K fields out, vacuum propagator once
    prof_end(tok, st, (8.0 + 8.0 * K) * plane * nb + 8.0 * plane);
    w.slice = s;
    w.last = (s == n_slices - 1);
    w.snap = stack ? stack + (long long)s * plane : nullptr;
    tok = prof_begin(WAP_KIND_WPM_ROW, st);
    if ((e = launch_wpm_row(p->nx, p->row_e, w, nb, rows, st)) != cudaSuccess) return cuda_fail(e, "wpm row pass");
    // K fields in, potential, wave out (+ dp buffer on the last slice, + snapshot)
    prof_end(tok, st, (8.0 * K + 4.0 + 8.0 + (w.last ? 8.0 : 0.0) + (w.snap ? 8.0 : 0.0)) * plane * nb);
    if (w.blend) {
      // row FFT of the blended wave; the spatial wave is this slice's snapshot
      // (at the last slice: the exit wave, the transform going to the dp buffer)
      fin.probe0 = b0;
      fin.psi = w.last ? p->dpbuf : exit;
      fin.psi_bstride = plane;
      fin.snap = w.last ? exit : w.snap;
      fin.snap_bstride = w.last ? plane : (long long)n_slices * plane;
      if ((e = launch_row(p->nx, p->row_e, fin, nb, rows, st)) != cudaSuccess) return cuda_fail(e, "wpm row FFT");
      if (w.last && w.snap &&
          (e = cudaMemcpy2DAsync(w.snap + (long long)b0 * n_slices * plane, (size_t)n_slices * plane * sizeof(float2),
                                 exit + (long long)b0 * plane, plane * sizeof(float2),
                                 plane * sizeof(float2), nb, cudaMemcpyDeviceToDevice, st)) != cudaSuccess)
        return cuda_fail(e, "wpm last snapshot");
    }
  }
  return WAP_OK;
}

}  // namespace wap

using namespace wap;

extern "C" int wap_wpm_fwd(wap_plan* p, const float* V, int n_slices, int n_draws, const int32_t* draw,
                           const float* psi0, int n_probes, int psi0_per_probe, const int32_t* positions, double dz,
                           double energy, double sampling_y, double sampling_x, double power_spacing, float* exit,
                           float* dp, float* stack, void* stream) {
  clear_error();
  int rc = check_common(p, V, n_slices, n_draws, psi0, n_probes, exit);
  if (rc) return rc;
  if (p->op != WAP_OP_WPM) return fail(WAP_ERR_ARG, "plan was not created for the WPM path");
  if (!(sampling_y > 0) || !(sampling_x > 0)) return fail(WAP_ERR_ARG, "sampling must be positive");
  if (!(power_spacing > 0)) return fail(WAP_ERR_ARG, "power_spacing must be positive");
  cudaStream_t st = (cudaStream_t)stream;
  const Physics ph = physics(energy, dz);
  const int K = p->n_bins;
  const long long plane = (long long)p->ny * p->nx;
  cudaError_t e;

  const double key[4] = {sampling_y, sampling_x, dz, energy};
  if (!std::equal(key, key + 4, p->hvac_key)) {
    HvacArgs h{p->ny, p->nx, sampling_y, sampling_x, dz, ph.k0, p->hvac, p->hvac_lo, p->ky2, p->kx2, p->q};
    count_launch();
    wpm_vacuum_kernel<<<(unsigned)((plane + 255) / 256), 256, 0, st>>>(h);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "wpm_vacuum_kernel");
    std::copy(key, key + 4, p->hvac_key);
  }
  WpmNodeScalars nodes;
  if ((rc = wpm_slices(p, V, n_slices, n_draws, ph, dz, sampling_y, sampling_x, power_spacing, &nodes, st))) return rc;
  // psi0 -> row spectrum
  RowArgs r = base_row_args(p, ph, V, n_slices, draw);
  r.psi = reinterpret_cast<float2*>(exit);
  r.psi_bstride = plane;
  r.src = reinterpret_cast<const float2*>(psi0);
  r.src_bstride = psi0_per_probe ? plane : 0;
  r.shifts = positions;
  r.flags = ROW_LOAD_SRC | ROW_FFT;
  if (!p->generic && (e = row_chunks(p, r, n_probes, st)) != cudaSuccess) return cuda_fail(e, "row pass");

  WpmColArgs c{};
  c.psi = reinterpret_cast<const float2*>(exit);
  c.fields = p->fields;
  c.hvac = p->hvac;
  c.hvac_lo = p->hvac_lo;
  c.ky2 = p->ky2;
  c.kx2 = p->kx2;
  c.q = p->q;
  c.refs = p->refs;
  c.draw = draw;
  c.tw = p->tw_col;
  c.ny = p->ny;
  c.nx = p->nx;
  c.K = K;
  c.n_slices = n_slices;
  c.k02 = (float)(ph.k0 * ph.k0);
  c.dz = (float)dz;
  c.det = p->det.resolved(p->ny, p->nx);

  WpmRowArgs w{};
  w.psi = reinterpret_cast<float2*>(exit);
  w.fields = p->fields;
  w.dpbuf = p->dpbuf;
  w.dpbuf_bstride = plane;
  w.V = V;
  w.draw = draw;
  w.v_draw_stride = (long long)n_slices * plane;
  w.refs = p->refs;
  w.tw = p->tw_row;
  w.ny = p->ny;
  w.nx = p->nx;
  w.K = K;
  w.n_slices = n_slices;
  w.scale = (float)(1.0 / (double)plane);
  w.ri_a = (float)ph.ri_a;
  w.ri_inv_den = (float)ph.ri_inv_den;
  w.snap_bstride = (long long)n_slices * plane;

  if (p->generic)
    return generic_wpm_forward(p, c, w, nodes, power_spacing, r.src, r.src_bstride, positions, n_slices, n_probes, dp,
                               reinterpret_cast<float2*>(stack), st);
  for (int b0 = 0; b0 < n_probes; b0 += 65535) {
    const int nb = std::min(65535, n_probes - b0);
    c.probe0 = b0;
    w.probe0 = b0;
    rc = nodes.nodes ? node_slices(p, nodes, c, w, power_spacing, n_slices, nb, reinterpret_cast<float2*>(stack), st)
                     : reference_slices(p, ph, V, draw, c, w, n_slices, b0, nb, reinterpret_cast<float2*>(exit),
                                        reinterpret_cast<float2*>(stack), st);
    if (rc) return rc;
    if (dp) {
      WpmColArgs d = c;
      d.psi = p->dpbuf;
      d.dp = dp;
      d.dp_mode = 1;
      const ProfToken tok = prof_begin(WAP_KIND_WPM_COL, st);
      if ((e = launch_wpm_col(p->ny, p->col_e, d, nb, p->col_w, st)) != cudaSuccess) return cuda_fail(e, "wpm dp pass");
      prof_end(tok, st, 12.0 * plane * nb);
    }
  }
  return WAP_OK;
}
