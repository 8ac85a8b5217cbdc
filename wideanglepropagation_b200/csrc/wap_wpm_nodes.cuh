// Wide-angle (WPM) slice step by interpolation over the reference index.
//
// The step needs, per pixel, two of the K reference fields
//   u(a) = ifft2(exp(i dz sqrt(q + a)) fft2(psi)),  q = k0^2 - k_perp^2,
//   a_k = k0^2 delta_k (2 + delta_k),
// (propagation.py:159-167, :239-254), and u depends on its index only through
// a, smoothly: exp(i dz (sqrt(q + a) - sqrt(q))) = exp(i kappa a) exp(i g(a; q))
// with kappa = dz / (2 sqrt(q)) taken midway over the grid, so that g is the
// small rest (the variation of 1 / sqrt(q) over the grid, and the curvature of
// the square root: ~1e-3 rad for light atoms at 300 keV).  The first factor
// is a number per pixel; the second is interpolated in a at r Chebyshev nodes
// of the slice's range:
//   u(a) = exp(i kappa a) sum_j l_j(tau(a)) G_j,   G_j = ifft2(exp(i g(a_j; q)) Hvac fft2(psi)).
// r is the smallest count whose remainder bound is below kWpmNodeTol for the
// slice's range of a (wpm_node_count): 2 to 5 for light to heavy atoms, whatever K is.
// The blend of the two bracketing references is unchanged, pixel by pixel; only
// the K inverse transforms become r (one 512^2 probe, 200 slices, K = 16: 11.7 ->
// 3.67 ms; 256^2, 40 slices, K = 128: 3.31 -> 0.47 ms).  A slice whose range has no
// such r < K, or reaches towards the evanescent edge, forms its K reference fields
// (nodes = 0 in its record).
//
// Fields are stored as the centre node's G_c and the differences G_j - G_c
// (|.| ~ 1e-3 |G_c|): sum_j l_j = 1, so u = exp(i kappa a) (G_c + sum l_j (G_j - G_c)),
// and the rounding of the r - 1 further transforms is scaled down with them.
#pragma once
#include "wap_passes.cuh"

namespace wap {

constexpr int kWpmMaxNodes = 12;
// absolute error of the interpolated factor exp(i g) (unit modulus) per slice:
// 200 slices add at most 2e-7 to a float32 rounding of ~1.5e-6 of the same chain
constexpr double kWpmNodeTol = 1.0e-9;

// What a slice's column and row passes need to know, written by wpm_slices_kernel.
struct WpmSlice {
  int nf;          // fields formed
  int nodes;       // 1: interpolation nodes (field 0 the centre node, the others differences); 0: the K references
  float xc;        // centre of the range of x = delta (2 + delta) = a / k0^2
  float inv_xh;    // 1 / half width (0: one point)
  float a0;        // a of field 0 (the centre node)
  float dlo;       // smallest delta of the slice, and 1 / (largest - smallest) (0: one value)
  float inv_range;
  float pad;
  float da[kWpmMaxNodes];    // a_j - a0 of field j
  float bw[kWpmMaxNodes];    // 1 / prod_{m != j} (tau_j - tau_m)
  float other[kWpmMaxNodes][kWpmMaxNodes];   // [j]: the nf - 1 node positions tau_m, m != j
};

// delta = sqrt(1 + r) - 1 of r = n^2 - 1: the series of the square root for
// |r| <= 1/64 (truncation 4e-11 of delta), where all but absurd potentials lie
__device__ __forceinline__ float wpm_delta(float r) {
  if (fabsf(r) <= 0.015625f)
    return r * fmaf(r, fmaf(r, fmaf(r, fmaf(r, 0.02734375f, -0.0390625f), 0.0625f), -0.125f), 0.5f);
  return r / (sqrtf(1.0f + r) + 1.0f);
}

// ---------------------------------------------------------------------------
// column side: the spectrum factors of the nodes
// ---------------------------------------------------------------------------
// exp(i x) - 1 without cancellation: the Taylor series of cis_small, and
// (-2 sin^2(x/2), sin x) for larger phases
static __device__ __noinline__ float2 cism1_large(float x) {
  float s, c, h, g;
  sincosf(x, &s, &c);
  sincosf(0.5f * x, &h, &g);
  return make_float2(-2.0f * h * h, s);
}
__device__ __forceinline__ float2 cism1(float x) {
  if (fabsf(x) > 0.5f) return cism1_large(x);
  const float p2 = x * x;
  const float sn = x * fmaf(p2, fmaf(p2, fmaf(p2, fmaf(p2, 2.7557319e-06f, -1.9841270e-04f), 8.3333333e-03f),
                                     -1.6666667e-01f), 1.0f);
  const float cm = p2 * fmaf(p2, fmaf(p2, fmaf(p2, fmaf(p2, -2.7557319e-07f, 2.4801587e-05f), -1.3888889e-03f),
                                      4.1666667e-02f), -0.5f);
  return make_float2(cm, sn);
}
// 1 / sqrt(q): the hardware's estimate and one Newton step
__device__ __forceinline__ float rsqrt_1ulp(float q) {
  const float p = rsqrtf(q);
  return fmaf(0.5f * p, fmaf(-q * p, p, 1.0f), p);
}
// Slope of dz sqrt(q) at q = qbar (1 - eps) less kappa, its value at qbar: with
// s = sqrt(q / qbar), kappa (1 / s - 1) = kappa eps / (s + s^2) - the difference of
// the two, with a rounding error of its own size and not of kappa's.
__device__ __forceinline__ float wpm_slope_rest(float q, float eps, float kappa, float inv_root_qbar) {
  const float s = q * rsqrt_1ulp(q) * inv_root_qbar;
  return __fdividef(kappa * eps, fmaf(s, s, s));
}
// dz (sqrt(q1 + da) - sqrt(q1)) / da - kappa for a step outside the series' range
static __device__ __noinline__ float wpm_mean_slope_direct(float s, float da, float dz) {
  const float r1 = 0.5f * dz / s;   // sqrt(q1), with the sign of dz
  return dz / (r1 + copysignf(sqrtf(fmaf(r1, r1, da)), r1));
}
// Mean slope of dz sqrt(q) between q1 and q1 + da less kappa, from the slope rest
// at q1: slope 2 / (1 + sqrt(1 + x)), x = da / q1 = da (2 slope / dz)^2, as its
// series (x^4 term below 1e-9 for |x| <= 1/128)
__device__ __forceinline__ float wpm_mean_slope(float rest, float kappa, float da, float dz, float c4) {
  const float s = kappa + rest, x = da * c4 * s * s;
  if (fabsf(x) <= 0.0078125f) return fmaf(s * x, fmaf(x, fmaf(x, -0.078125f, 0.125f), -0.25f), rest);
  return wpm_mean_slope_direct(s, da, dz) - kappa;
}

struct WpmNodeColArgs {
  WpmColArgs c;              // as the reference-field kernel (tw: the (ny, 8) table; kpg unused)
  const WpmSlice* rec;
  float kappa;               // dz / (2 sqrt(qbar))
  float dq, inv_qbar, inv_root_qbar;   // qbar - k0^2, 1 / qbar, 1 / sqrt(qbar)
  float c4;                  // 4 / dz^2
  bool sharing;              // launch only: slices without nodes may be shared out (SPLIT)
};

// Barrier of one group of threads of a block (whole warps).
__device__ __forceinline__ void group_sync(int bar, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory");
}

// Column exchange of one group: its own [N][w] tile and barrier.
struct GroupColExchange {
  float2* base;
  int w, c, bar, threads;
  __device__ __forceinline__ void st(int p, float2 v) const { base[p * w + c] = v; }
  __device__ __forceinline__ float2 ld(int p) const { return base[p * w + c]; }
  __device__ __forceinline__ void st2(int b, int o, float2 v) const { st(b + o, v); }
  __device__ __forceinline__ float2 ld2(int b, int o) const { return ld(b + o); }
  __device__ __forceinline__ void sync() const { group_sync(bar, threads); }
};

// Groups per line (G of the kernels below) when few lines are in flight.
__host__ __device__ constexpr int node_col_groups(int n) { return n >= 2048 ? 1 : 2; }
__host__ __device__ constexpr int node_row_groups(int n) { return n >= 2048 ? 1 : n >= 1024 ? 2 : 4; }
// Threads and resident blocks of the column pass.  At 1024 points 512 threads hold
// four columns, twice per SM (one 1024^2 probe, 40 slices: 3.09 ms with one block of
// 128 registers per thread, 3.02 with two of 64), or two columns in two groups (1024 x
// 256: 1.27 ms as one block of 1024 threads, 0.92 now).
__host__ __device__ constexpr int node_col_threads(int n, int g) {
  return n >= 2048 ? 512 * g : n >= 1024 ? 512 : 256 * g;
}
__host__ __device__ constexpr int node_col_blocks(int n, int g) { return g > 1 || n >= 2048 ? 1 : n >= 1024 ? 2 : 3; }

// Column pass: column FFT, * Hvac * exp(i g(a0; q)), then per field its factor
// and the inverse column FFT.  With G groups of threads per column tile, group 0
// does the forward part and hands the spectrum over through shared memory, and
// group g takes the fields g, g + G, ...: few probes fill few warps, and a
// warp's chain of transforms is what the pass waits for.
//
// The column k_x = 0 of a plane wave is nearly constant, and its whole intensity
// passes through one number, the sum over the column, whose roundings (the last
// additions, the factor, the first additions back) no averaging reduces.  That
// column is transformed less its first element; the constant part, one number
// for the whole column, is propagated beside it in float64 and added to the
// results, row by row.  Drift of |psi| over 200 slices of 512^2, rms over
// specimens: 5.9e-7 without, 4.1e-8 with (the exit wave's error 2.0e-6, 1.5e-6).
//
// SPLIT: a slice without nodes shares its K fields out to the blocks of grid.z too,
// each of which repeats the forward part; a slice with nodes leaves them at once.
template <int NY, int E, int G, bool SPLIT>
__global__ void __launch_bounds__(node_col_threads(NY, G), node_col_blocks(NY, G))
wpm_node_col_kernel(const WpmNodeColArgs na) {
  using P = FFTPlan<NY, E>;
  constexpr int T = P::T;
  const WpmColArgs& a = na.c;
  const int group = blockDim.x / G;      // threads of one group
  const int W = group / T;
  extern __shared__ float4 smem_raw[];
  float4* tw = smem_raw;
  const int g = G == 1 ? 0 : threadIdx.x / group;
  const int gt = threadIdx.x - g * group;
  const int c = gt & (W - 1);
  const int t = gt / W;
  const int col = blockIdx.x * W + c;
  const int b = a.probe0 + blockIdx.y;
  const int nx = a.nx, step = T * nx;
  const int first = t * nx + col;        // element e of this thread: first + e step
  const int plane = NY * nx;
  float2* tiles = reinterpret_cast<float2*>(tw + P::TW_SIZE);
  const GroupColExchange xs{tiles + g * NY * W, W, c, 1 + g, group};
  // nothing here depends on the previous pass: twiddles and the slice's record
  // are read under its tail
  if constexpr (!SPLIT)
    for (int i = threadIdx.x; i < P::TW_SIZE; i += blockDim.x) tw[i] = __ldg(a.tw + i);
  const int d = a.draw ? a.draw[b] : 0;
  const long long srow = (long long)d * a.n_slices + a.slice;
  const WpmSlice* rec = na.rec + srow;
  if constexpr (SPLIT) {
    if (blockIdx.z > 0 && rec->nodes) return;
    for (int i = threadIdx.x; i < P::TW_SIZE; i += blockDim.x) tw[i] = __ldg(a.tw + i);
  }
  const int nf = rec->nf;
  const bool nodes = rec->nodes != 0;
  const float a0 = rec->a0;   // 0 without nodes
  // slope rest at q + a0 of this thread's elements; without nodes the slope at q
  // (0 beyond the evanescent edge)
  const float kx2 = __ldg(a.kx2 + col);
  float p[E];
  if (nodes) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float k2 = __ldg(a.ky2 + t + T * e) + kx2;
      p[e] = wpm_slope_rest(a.k02 + a0 - k2, (na.dq - a0 + k2) * na.inv_qbar, na.kappa, na.inv_root_qbar);
    }
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float q = __ldg(a.q + first + e * step);
      p[e] = q > 0.0f ? 0.5f * a.dz * sqrtf(1.0f / q) : 0.0f;
    }
  }
  __syncthreads();
  pdl_wait_then_release();
  const bool apart = blockIdx.x == 0 && nodes;   // this block holds the column k_x = 0
  const float2 ref = apart && col == 0 ? __ldcg(a.psi + (long long)b * plane) : make_float2(0.f, 0.f);
  float2 v[E];
  if (g == 0) {
    const float2* pcol = a.psi + (long long)b * plane + first;
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = __ldcg(pcol + e * step);
    if (apart) {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = csub(v[e], ref);
    }
    fft<NY, E, false>(v, t, xs, tw);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int o = first + e * step;
      const float2 h = __ldg(a.hvac + o);
      float2 l = __ldg(a.hvac_lo + o);
      // Hvac (1 + m) as Hvac's hi part and a small rest: one rounding of the wave for
      // both factors (the slope taken from q + a0 back to q; a0 = 0 without nodes)
      if (nodes) {
        const float2 m = cism1(a0 * wpm_mean_slope(p[e], na.kappa, -a0, a.dz, na.c4));
        l = make_float2(fmaf(h.x, m.x, fmaf(-h.y, m.y, l.x)), fmaf(h.x, m.y, fmaf(h.y, m.x, l.y)));
      }
      v[e] = cmul_hl(v[e], h, l);
    }
    if constexpr (G > 1) {
      xs.sync();
#pragma unroll
      for (int e = 0; e < E; ++e) xs.st(t + T * e, v[e]);
    }
  }
  if constexpr (G > 1) {
    __syncthreads();
    if (g > 0) {
      const GroupColExchange x0{tiles, W, c, 0, 0};
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = x0.ld(t + T * e);
    }
    __syncthreads();   // group 0 may overwrite its tile
  }
  // the constant part times the factor of (k_y = 0, this column) and n_y
  float2 ch = make_float2(0.f, 0.f), cl = ch;
  float rest0 = 0.f;
  if (apart) {
    const float k2 = __ldg(a.ky2) + kx2;
    rest0 = wpm_slope_rest(a.k02 + a0 - k2, (na.dq - a0 + k2) * na.inv_qbar, na.kappa, na.inv_root_qbar);
    const float2 m = cism1(a0 * wpm_mean_slope(rest0, na.kappa, -a0, a.dz, na.c4));
    const float2 h = __ldg(a.hvac + col), l = __ldg(a.hvac_lo + col);
    const double hx = (double)h.x + (h.x * m.x - h.y * m.y + l.x), hy = (double)h.y + (h.x * m.y + h.y * m.x + l.y);
    const double cx = NY * (ref.x * hx - ref.y * hy), cy = NY * (ref.x * hy + ref.y * hx);
    ch = make_float2((float)cx, (float)cy);
    cl = make_float2((float)(cx - ch.x), (float)(cy - ch.y));
  }
  float2* fcol = a.fields + (long long)b * a.K * plane + first;
  const float* refs = a.refs + srow * a.K;
  const int shares = SPLIT && !nodes ? gridDim.z : 1;
  for (int k = SPLIT ? blockIdx.z * G + g : g; k < nf; k += G * shares) {
    float2 u[E];
    if (nodes) {
      if (k == 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) u[e] = v[e];
      } else {
        const float da = rec->da[k];
#pragma unroll
        for (int e = 0; e < E; ++e) u[e] = cmul(v[e], cism1(da * wpm_mean_slope(p[e], na.kappa, da, a.dz, na.c4)));
      }
    } else {
      const float dk = refs[k];
      const float ak = a.k02 * dk * (2.0f + dk);   // n_k^2 k0^2 - k0^2
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float x = ak * na.c4 * p[e] * p[e];   // a_k / q
        if (p[e] != 0.0f && fabsf(x) <= 0.0078125f)
          u[e] = cmul(v[e], cis_small(ak * p[e] * fmaf(x, fmaf(x, fmaf(x, -0.078125f, 0.125f), -0.25f), 1.0f)));
        else
          u[e] = wpm_bin_direct(v[e], 1.0f / __ldg(a.q + first + e * step), ak, a.dz, a.hvac + first + e * step);
      }
    }
    fft<NY, E, true>(u, t, xs, tw);
    if (apart) {
      float2 hi = ch, lo = cl;
      if (k > 0) {
        const float da = rec->da[k];
        hi = cmul(ch, cism1(da * wpm_mean_slope(rest0, na.kappa, da, a.dz, na.c4)));
        lo = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int e = 0; e < E; ++e) u[e] = cadd(cadd(u[e], lo), hi);
    }
    float2* fk = fcol + (long long)k * plane;
#pragma unroll
    for (int e = 0; e < E; ++e) __stcg(fk + e * step, u[e]);
  }
}

// ---------------------------------------------------------------------------
// row side: the pixels' weights
// ---------------------------------------------------------------------------
// A pixel's blend of its two bracketing references (searchsorted(left),
// clip(1, K - 1), smoothstep: propagation.py:239-249): the weight w of the right
// one, exp(i kappa a) - 1 of each times its weight (pl, pr), and their places
// tl, tr: tau of the references (nodes) or the left reference's number (as int
// bits in tl; pl, pr unused).
struct WpmPixel {
  float2 pl, pr;
  float w, tl, tr;
};

// First index with refs[i] >= dn.  Evenly spaced references (power 1) and
// quadratic ones (power 2, the default) are found from the pixel's place in the
// range, put right by comparing with the references beside it (two reads where a
// binary search takes log2 K); other spacings by binary search.
__device__ __forceinline__ int wpm_search(const float* srefs, int K, float dn, float dlo, float inv_range, int spacing) {
  if (spacing == 0) {
    int lo = 0, hi = K;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (srefs[mid] < dn) lo = mid + 1; else hi = mid;
    }
    return lo;
  }
  float f = (dn - dlo) * inv_range;
  f = fminf(fmaxf(f, 0.0f), 1.0f);   // 0 for a NaN
  if (spacing == 2) f = sqrtf(f);
  int i = (int)(f * (float)(K - 1));
  while (i > 0 && srefs[i - 1] >= dn) --i;
  while (i < K && srefs[i] < dn) ++i;
  return i;
}

__device__ __forceinline__ WpmPixel wpm_pixel(float volts, const float* srefs, int K, float ri_a, float ri_inv_den,
                                              const WpmSlice& rec, int spacing, float2 kk) {
  const float dn = wpm_delta(volts * (ri_a + volts) * ri_inv_den);
  const int ir = min(max(wpm_search(srefs, K, dn, rec.dlo, rec.inv_range, spacing), 1), K - 1);
  const float nl = srefs[ir - 1], nr = srefs[ir];
  const float den = nr - nl;
  // (an IEEE division here leaves the error of a step against float64 where it is,
  // 1.700e-7 at K = 4 over a range of 400 V, and costs 1.4 % of a 512^2 call)
  float w = __fdividef(dn - nl, den == 0.0f ? 1.0f : den);
  w = fminf(fmaxf(w, 0.0f), 1.0f);
  w = w * w * (3.0f - 2.0f * w);
  WpmPixel p;
  p.w = w;
  if (rec.nodes) {
    // kappa a = kappa k0^2 x with the constant as hi + lo: its rounding would scale
    // the potential alike in every slice
    const float xl = nl * (2.0f + nl), xr = nr * (2.0f + nr);
    p.pl = cscale(cism1(fmaf(xl, kk.x, xl * kk.y)), 1.0f - w);
    p.pr = cscale(cism1(fmaf(xr, kk.x, xr * kk.y)), w);
    p.tl = fminf(fmaxf((xl - rec.xc) * rec.inv_xh, -1.0f), 1.0f);
    p.tr = fminf(fmaxf((xr - rec.xc) * rec.inv_xh, -1.0f), 1.0f);
  } else {
    p.pl = p.pr = make_float2(0.f, 0.f);
    p.tl = __int_as_float(ir - 1);
    p.tr = 0.f;
  }
  return p;
}

struct WpmNodeRowArgs {
  WpmRowArgs r;              // as the reference-field kernel (tw: the (nx, 8) table; kpg: bins of a SPLIT share)
  const WpmSlice* rec;
  unsigned* tiles;           // SPLIT: shares of each row tile that are done (zero between passes)
  float2 kk;                 // kappa k0^2, hi and lo parts
  int spacing;               // 1, 2: the references' power; 0: another
  bool sharing;              // as WpmNodeColArgs::sharing
};

// Row exchange of one row of one group: its own segment, synchronised by the
// warp (T <= 32) or by named barrier `bar` over the row's T threads.
template <int T>
struct GroupRowExchange {
  float2* base;
  int bar;
  __device__ __forceinline__ void st(int p, float2 v) const { base[p + (p >> 4)] = v; }
  __device__ __forceinline__ float2 ld(int p) const { return base[p + (p >> 4)]; }
  __device__ __forceinline__ void st2(int b, int o, float2 v) const { st(b + o, v); }
  __device__ __forceinline__ float2 ld2(int b, int o) const { return ld(b + o); }
  __device__ __forceinline__ void sync() const {
    if constexpr (T <= 32) __syncwarp();
    else group_sync(bar, T);
  }
};

// Row pass: per field its inverse row FFT, the weighted sum, the row FFT of the
// next slice.  With G groups of threads per row tile, group g transforms the
// fields g, g + G, ... and adds up its share of the blend; group 0 folds the
// shares through shared memory and goes on alone (as in the column pass).
// The pixels' blends depend on the potential alone: the groups form them
// together, before the wait for the column pass, and leave them in shared memory.
//
// SPLIT: a slice without nodes shares its bins out to the blocks of grid.z too, as in
// wpm_row_kernel: block z owns the pixels whose left bin lies in [z kpg, z kpg + kpg),
// passes over the bins that none of them wants, and stores their blend; the block of a
// tile that is done last (a count per tile) takes the whole row on.  One 256^2 probe, K =
// 128, 20 slices that have no nodes: 4.67 -> 2.01 ms (2.07 by the reference-field kernels).
template <int NX, int E, int G, bool SPLIT>
__global__ void __launch_bounds__(kRowThreads * (G > 1 ? 2 : 1), G > 1 ? 2 : 3)
wpm_node_row_kernel(const WpmNodeRowArgs na) {
  using C = RowCfg<NX, E>;
  constexpr int T = C::T;
  const WpmRowArgs& a = na.r;
  const int group = blockDim.x / G;
  const int rows = group / T;
  extern __shared__ float4 smem_raw[];
  float4* tw = smem_raw;
  float4* spw = tw + C::P::TW_SIZE;                                   // (pl, pr) of a pixel
  float2* spt = reinterpret_cast<float2*>(spw + rows * NX);           // (tl, tr)
  float2* xbuf = spt + rows * NX;
  float* sw = reinterpret_cast<float*>(xbuf + rows * G * C::PADN);    // w
  float* srefs = sw + rows * NX;
  __shared__ WpmSlice srec;
  const int b = a.probe0 + blockIdx.y;
  const int d = a.draw ? a.draw[b] : 0;
  const long long srow = (long long)d * a.n_slices + a.slice;
  const int g = G == 1 ? 0 : threadIdx.x / group;
  const int rl = (threadIdx.x - g * group) / T;
  const int t = threadIdx.x & (T - 1);
  const int row = blockIdx.x * rows + rl;
  const int plane = a.ny * NX, at = row * NX + t;
  if constexpr (SPLIT) {
    if (blockIdx.z > 0 && (na.rec + srow)->nodes) return;
  }
  __shared__ unsigned used[SPLIT ? 128 : 1];   // bins (n_bins <= 4096) that this block's pixels want
  __shared__ int last_share;
  const float* vrow = a.V + (long long)d * a.v_draw_stride + (long long)a.slice * plane + at;
  float vv[E / G];
#pragma unroll
  for (int i = 0; i < E / G; ++i) vv[i] = __ldg(vrow + T * (g + G * i));
  for (int i = threadIdx.x; i < C::P::TW_SIZE; i += blockDim.x) tw[i] = __ldg(a.tw + i);
  for (int i = threadIdx.x; i < a.K; i += blockDim.x) srefs[i] = __ldg(a.refs + srow * a.K + i);
  for (int i = threadIdx.x; i < (int)(sizeof(WpmSlice) / 4); i += blockDim.x)
    reinterpret_cast<int*>(&srec)[i] = __ldg(reinterpret_cast<const int*>(na.rec + srow) + i);
  if constexpr (SPLIT)
    for (int i = threadIdx.x; i < 128; i += blockDim.x) used[i] = 0u;
  __syncthreads();
  const bool nodes = srec.nodes != 0;
  const int nf = srec.nf;
  const bool split = SPLIT && !nodes;
  const int kb = split ? blockIdx.z * a.kpg : 0, kl = split ? min(kb + a.kpg, a.K - 1) : 0;   // owned left bins
  spw += rl * NX;
  spt += rl * NX;
  sw += rl * NX;
#pragma unroll
  for (int i = 0; i < E / G; ++i) {
    const WpmPixel px = wpm_pixel(vv[i], srefs, a.K, a.ri_a, a.ri_inv_den, srec, na.spacing, na.kk);
    const int x = t + T * (g + G * i);
    spw[x] = make_float4(px.pl.x, px.pl.y, px.pr.x, px.pr.y);
    spt[x] = make_float2(px.tl, px.tr);
    sw[x] = px.w;
    if (SPLIT && split) {
      const int il = __float_as_int(px.tl);
      if (il >= kb && il < kl) {
        atomicOr(used + (il >> 5), 1u << (il & 31));
        atomicOr(used + ((il + 1) >> 5), 1u << ((il + 1) & 31));
      }
    }
  }
  __syncthreads();
  pdl_wait_then_release();

  // acc: the differences' share of the blend (or, without nodes, the blend).  The
  // centre field comes last and meets the sum of all shares in one addition: of
  // the full-sized values only that one is rounded here.
  float2 acc[E], u[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = make_float2(0.f, 0.f);
  const GroupRowExchange<T> xs{xbuf + (g * rows + rl) * C::PADN, 1 + g * rows + rl};
  const float2* frow = a.fields + (long long)b * a.K * plane + at;
  const int n = split ? kl - kb + 1 : nf;   // fields of this block, from kb on
  for (int i = g < n ? g + (n - 1 - g) / G * G : -1; i >= 0; i -= G) {
    const int k = SPLIT ? kb + i : i;
    if (SPLIT && split && !(used[k >> 5] & (1u << (k & 31)))) continue;
    const float2* fk = frow + (long long)k * plane;
#pragma unroll
    for (int e = 0; e < E; ++e) u[e] = __ldcg(fk + T * e);
    fft<NX, E, true>(u, t, xs, tw);
    if (!nodes) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int il = __float_as_int(spt[t + T * e].x);
        const float w = il == k ? 1.0f - sw[t + T * e] : (il + 1 == k ? sw[t + T * e] : 0.0f);
        acc[e] = make_float2(fmaf(w, u[e].x, acc[e].x), fmaf(w, u[e].y, acc[e].y));
      }
    } else if (k > 0) {
      // l_k(tl), l_k(tr) of the pixels
      float wl[E], wr[E];
#pragma unroll
      for (int e = 0; e < E; ++e) wl[e] = wr[e] = srec.bw[k];
      for (int m = 0; m < nf - 1; ++m) {
        const float tm = srec.other[k][m];
#pragma unroll
        for (int e = 0; e < E; ++e) {
          const float2 p = spt[t + T * e];
          wl[e] *= p.x - tm;
          wr[e] *= p.y - tm;
        }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float4 m = spw[t + T * e];
        const float s = sw[t + T * e];
        const float wx = fmaf(wl[e], 1.0f - s + m.x, wr[e] * (s + m.z)), wy = fmaf(wl[e], m.y, wr[e] * m.w);
        acc[e] = make_float2(fmaf(wx, u[e].x, fmaf(-wy, u[e].y, acc[e].x)),
                             fmaf(wx, u[e].y, fmaf(wy, u[e].x, acc[e].y)));
      }
    }
  }
  if constexpr (G > 1) {
    if (g > 0) {
      xs.sync();   // the row's last exchange has been read
#pragma unroll
      for (int e = 0; e < E; ++e) xs.st(t + T * e, acc[e]);
    }
    __syncthreads();
    if (g > 0) return;
    const int shares = min(G, n);
    for (int h = 1; h < shares; ++h) {
      const GroupRowExchange<T> xh{xbuf + (h * rows + rl) * C::PADN, 0};
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] = cadd(acc[e], xh.ld(t + T * e));
    }
  }
  if (nodes) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float4 m = spw[t + T * e];
      const float mx = m.x + m.z, my = m.y + m.w;
      acc[e] = make_float2(u[e].x + fmaf(u[e].x, mx, fmaf(-u[e].y, my, acc[e].x)),
                           u[e].y + fmaf(u[e].x, my, fmaf(u[e].y, mx, acc[e].y)));
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = cscale(acc[e], a.scale);

  if (SPLIT && split && gridDim.z > 1) {
    float2* brow = a.blend + (long long)b * plane + at;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int il = __float_as_int(spt[t + T * e].x);
      if (il >= kb && il < kl) __stcg(brow + T * e, acc[e]);
    }
    __threadfence();
    group_sync(15, group);   // (group 0 is what is left of the block)
    if (threadIdx.x == 0) {
      unsigned* done = na.tiles + (long long)blockIdx.y * gridDim.x + blockIdx.x;
      last_share = atomicAdd(done, 1u) == gridDim.z - 1;
      if (last_share) *done = 0u;
      __threadfence();
    }
    group_sync(15, group);
    if (!last_share) return;
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = __ldcg(brow + T * e);
  }

  if (a.snap) {
    float2* sp = a.snap + (long long)b * a.snap_bstride + at;
#pragma unroll
    for (int e = 0; e < E; ++e) __stcs(sp + T * e, acc[e]);
  }
  float2* prow = a.psi + (long long)b * plane + at;
  if (a.last) {
#pragma unroll
    for (int e = 0; e < E; ++e) __stcg(prow + T * e, acc[e]);
  }
  fft<NX, E, false>(acc, t, xs, tw);
  float2* orow = a.last ? a.dpbuf + (long long)b * a.dpbuf_bstride + at : prow;
#pragma unroll
  for (int e = 0; e < E; ++e) __stcg(orow + T * e, acc[e]);
}

}  // namespace wap
