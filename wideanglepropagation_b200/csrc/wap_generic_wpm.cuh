// WPM on grids whose sides are not powers of two: the fields of a slice and their
// blend (wap_wpm_nodes.cuh has the method), whatever transforms the lines: the
// mixed-radix lines of wap_mixed.cuh (wap_generic_wpm.cu) or, along sides with a
// prime factor above 7, Bluestein's convolution (wap_bluestein.cu).
//
// The kernels take the line kind L: threads of a line, its twiddles, the values its
// exchanges hold along columns and rows, and pass(): one DFT of the line that `op`
// loads and stores (every thread of the block calls it; `live` lines only do work).
#pragma once
#include "wap_generic.cuh"
#include "wap_wpm_nodes.cuh"

namespace wap {

struct GenWpmColArgs {
  WpmNodeColArgs n;           // c.tw, c.kpg unused
  GenAxis ax;
  int w;                      // columns per block
  bool refs;                  // every slice forms its reference fields
};

struct GenWpmSpectrum {       // column DFT -> spectrum * Hvac (* the centre node's factor), or the pattern
  const WpmNodeColArgs& na;
  const float2* pcol;
  const float2* hvac;
  const float2* hvac_lo;
  float2* spec;               // this column's spectrum, stride w
  float* dp;
  float2 ref;                 // taken off the column k_x = 0 (0 elsewhere)
  float kx2, a0;
  int drx, w;
  bool nodes;
  __device__ __forceinline__ float2 load(int p) const { return csub(__ldcg(pcol + p * na.c.nx), ref); }
  __device__ __forceinline__ float2 turn(int, float2 y) const { return y; }
  __device__ __forceinline__ void store(int p, float2 y) const {
    if (dp) {
      gen_pattern(dp, na.c.det, drx, p, na.c.ny, y);
      return;
    }
    const int o = p * na.c.nx;
    const float2 h = __ldg(hvac + o);
    float2 l = __ldg(hvac_lo + o);
    if (nodes) {
      const float k2 = __ldg(na.c.ky2 + p) + kx2;
      const float rest = wpm_slope_rest(na.c.k02 + a0 - k2, (na.dq - a0 + k2) * na.inv_qbar, na.kappa, na.inv_root_qbar);
      const float2 m = cism1(a0 * wpm_mean_slope(rest, na.kappa, -a0, na.c.dz, na.c4));
      l = make_float2(fmaf(h.x, m.x, fmaf(-h.y, m.y, l.x)), fmaf(h.x, m.y, fmaf(h.y, m.x, l.y)));
    }
    spec[p * w] = cmul_hl(y, h, l);
  }
};

// a reference field's factor on one element: the series of the column passes, or the
// direct formulas near and beyond the edge
__device__ __forceinline__ float2 gen_reference_value(float2 u, float q, float ak, float dz, const float2* hvac) {
  const float pr = 1.0f / q, x = ak * pr;
  if (q > 0.0f && fabsf(x) <= 0.0078125f)
    return cmul(u, cis_small(ak * (0.5f * dz * sqrtf(pr)) *
                             fmaf(x, fmaf(x, fmaf(x, -0.078125f, 0.125f), -0.25f), 1.0f)));
  return wpm_bin_direct(u, pr, ak, dz, hvac);
}
// out of line in the instance whose slices mostly have nodes: one copy per kernel, not
// one per radix, and no registers of theirs
static __device__ __noinline__ float2 gen_reference_call(float2 u, float q, float ak, float dz, const float2* hvac) {
  return gen_reference_value(u, q, ak, dz, hvac);
}

template <bool REFS>
struct GenWpmField {          // spectrum * the field's factor -> inverse column DFT
  const WpmNodeColArgs& na;
  const float2* hvac;
  const float2* spec;
  float2* fcol;
  float2 ch, cl;              // the part taken off, propagated: added to every row
  float kx2, a0, da;          // da: a_k of a reference field
  int w, k;
  bool nodes;
  __device__ __forceinline__ float2 load(int p) const {
    const WpmColArgs& a = na.c;
    float2 u = spec[p * w];
    if (nodes) {
      if (k > 0) {
        const float k2 = __ldg(a.ky2 + p) + kx2;
        const float rest = wpm_slope_rest(a.k02 + a0 - k2, (na.dq - a0 + k2) * na.inv_qbar, na.kappa, na.inv_root_qbar);
        u = cmul(u, cism1(da * wpm_mean_slope(rest, na.kappa, da, a.dz, na.c4)));
      }
    } else {
      const float2* h = hvac + p * a.nx;
      const float q = __ldg(a.q + (h - a.hvac));
      u = REFS ? gen_reference_value(u, q, da, a.dz, h) : gen_reference_call(u, q, da, a.dz, h);
    }
    return cconj(u);
  }
  __device__ __forceinline__ float2 turn(int, float2 y) const { return y; }
  __device__ __forceinline__ void store(int p, float2 y) const {
    __stcg(fcol + p * na.c.nx, cadd(cadd(cconj(y), cl), ch));
  }
};

// Block group z forms the fields z, z + gridDim.z, ... (each repeats the forward
// transform: a column pass of one probe is a few dozen blocks).  REFS: the instance of
// grids that reach the evanescent edge, where every slice forms its reference fields.
template <class L, bool REFS>
__global__ void __launch_bounds__(L::kCol, L::kColBlocks) gen_wpm_col_kernel(const GenWpmColArgs ga) {
  extern __shared__ float4 gen_smem[];
  const GenAxis& ax = ga.ax;
  const WpmNodeColArgs& na = ga.n;
  const WpmColArgs& a = na.c;
  float4* tw = gen_smem;
  float2* bufs = reinterpret_cast<float2*>(tw + L::tw_len(ax));
  const int w = ga.w, c = threadIdx.x & (w - 1), t = threadIdx.x / w;
  float2* spec = bufs + L::col_len(ax) * w + c;
  for (int i = threadIdx.x; i < L::tw_len(ax); i += blockDim.x) tw[i] = __ldg(L::twiddles(ax) + i);
  const int col = blockIdx.x * w + c;
  const bool live = t < L::threads(ax) && col < a.nx;
  const int at = live ? col : 0;
  const int b = a.probe0 + blockIdx.y;
  const long long plane = (long long)a.ny * a.nx;
  const int d = a.draw ? a.draw[b] : 0;
  const long long srow = (long long)d * a.n_slices + a.slice;
  const WpmSlice* rec = na.rec + srow;
  const int nf = rec->nf;
  const bool nodes = !REFS && rec->nodes != 0;

  const auto mem = L::col_mem(ax, bufs, w, c);
  GenWpmSpectrum fwd{na};
  fwd.pcol = a.psi + (long long)b * plane + at;
  fwd.hvac = a.hvac + at;
  fwd.hvac_lo = a.hvac_lo + at;
  fwd.spec = spec;
  fwd.dp = a.dp_mode ? a.dp + (long long)b * a.det.plane() : nullptr;
  fwd.kx2 = __ldg(a.kx2 + at);
  fwd.a0 = rec->a0;
  fwd.drx = shifted(at, a.nx) - a.det.x0;
  fwd.w = w;
  fwd.nodes = nodes;
  __syncthreads();
  pdl_wait_then_release();
  if (!a.dp_mode && (int)blockIdx.z >= nf) return;
  // the column k_x = 0 less its first element, whose share is propagated beside it
  // (wpm_node_col_kernel)
  const bool apart = nodes && !a.dp_mode && live && col == 0;
  fwd.ref = apart ? __ldcg(a.psi + (long long)b * plane) : make_float2(0.f, 0.f);
  L::pass(ax, tw, mem, t, live, fwd);
  if (a.dp_mode) return;
  GenWpmField<REFS> inv{na};
  inv.hvac = fwd.hvac;
  inv.spec = spec;
  inv.kx2 = fwd.kx2;
  inv.a0 = fwd.a0;
  inv.w = w;
  inv.nodes = nodes;
  float2 ch = make_float2(0.f, 0.f), cl = ch;
  float rest0 = 0.f;
  if (apart) {
    const float k2 = __ldg(a.ky2) + fwd.kx2, a0 = fwd.a0;
    rest0 = wpm_slope_rest(a.k02 + a0 - k2, (na.dq - a0 + k2) * na.inv_qbar, na.kappa, na.inv_root_qbar);
    const float2 m = cism1(a0 * wpm_mean_slope(rest0, na.kappa, -a0, a.dz, na.c4));
    const float2 h = __ldg(fwd.hvac), l = __ldg(fwd.hvac_lo), r = fwd.ref;
    const double hx = (double)h.x + (h.x * m.x - h.y * m.y + l.x), hy = (double)h.y + (h.x * m.y + h.y * m.x + l.y);
    const double cx = a.ny * (r.x * hx - r.y * hy), cy = a.ny * (r.x * hy + r.y * hx);
    ch = make_float2((float)cx, (float)cy);
    cl = make_float2((float)(cx - ch.x), (float)(cy - ch.y));
  }
  for (int k = blockIdx.z; k < nf; k += gridDim.z) {
    __syncthreads();   // the spectrum is complete, and the last pass's buffers are free
    inv.k = k;
    inv.ch = ch;
    inv.cl = cl;
    if (nodes) {
      inv.da = rec->da[k];
      if (apart && k > 0) {
        inv.ch = cmul(ch, cism1(inv.da * wpm_mean_slope(rest0, na.kappa, inv.da, a.dz, na.c4)));
        inv.cl = make_float2(0.f, 0.f);
      }
    } else {
      const float dk = a.refs[srow * a.K + k];
      inv.da = a.k02 * dk * (2.0f + dk);   // n_k^2 k0^2 - k0^2
    }
    inv.fcol = a.fields + ((long long)b * a.K + k) * plane + at;
    L::pass(ax, tw, mem, t, live, inv);
  }
}

struct GenWpmRowArgs {
  WpmNodeRowArgs n;           // r.tw unused
  GenAxis ax;
  float2 scale;               // 1/(ny nx), hi + lo
  int rows;                   // per block
  int groups;                 // thread groups of a row (fields g, g + groups, ...)
};

struct GenWpmBlend {          // field -> inverse row DFT -> its share of the blend
  const float2* fk;
  const float4* spw;
  const float2* spt;
  const float* sw;
  const WpmSlice& rec;
  float2* acc;                // this group's share
  float2* centre;             // the centre field
  int k;
  bool nodes;
  __device__ __forceinline__ float2 load(int p) const { return cconj(__ldcg(fk + p)); }
  __device__ __forceinline__ float2 turn(int, float2 y) const { return y; }
  __device__ __forceinline__ void store(int p, float2 y) const {
    y = cconj(y);
    if (nodes && k == 0) {
      centre[p] = y;
      return;
    }
    const float2 pt = spt[p];
    const float s = sw[p];
    const float2 o = acc[p];
    if (!nodes) {
      const int il = __float_as_int(pt.x);
      const float wk = il == k ? 1.0f - s : (il + 1 == k ? s : 0.0f);
      acc[p] = make_float2(fmaf(wk, y.x, o.x), fmaf(wk, y.y, o.y));
      return;
    }
    const float4 m = spw[p];
    float wl = rec.bw[k], wr = wl;
    for (int i = 0; i < rec.nf - 1; ++i) {
      wl *= pt.x - rec.other[k][i];
      wr *= pt.y - rec.other[k][i];
    }
    const float wx = fmaf(wl, 1.0f - s + m.x, wr * (s + m.z)), wy = fmaf(wl, m.y, wr * m.w);
    acc[p] = make_float2(fmaf(wx, y.x, fmaf(-wy, y.y, o.x)), fmaf(wx, y.y, fmaf(wy, y.x, o.y)));
  }
};

struct GenWpmNext {           // blended wave -> row DFT of the next slice
  const float2* wave;
  float2* orow;
  __device__ __forceinline__ float2 load(int p) const { return wave[p]; }
  __device__ __forceinline__ float2 turn(int, float2 y) const { return y; }
  __device__ __forceinline__ void store(int p, float2 y) const { __stcg(orow + p, y); }
};

// Group g of a row transforms the fields g, g + G, ... and adds up its share of the
// blend; then the whole block adds the shares to the centre field and group 0
// transforms the sum.  The pixels' blends are formed before the wait for the
// column pass.
template <class L>
__global__ void __launch_bounds__(2 * kGenThreads) gen_wpm_row_kernel(const GenWpmRowArgs ga) {
  extern __shared__ float4 gen_smem[];
  __shared__ WpmSlice srec;
  const GenAxis& ax = ga.ax;
  const WpmNodeRowArgs& na = ga.n;
  const WpmRowArgs& a = na.r;
  const int T = L::threads(ax), G = ga.groups, rows = ga.rows, n = a.nx;
  // twiddles, (pl, pr), (tl, tr), transform buffers, shares, centre field, w, references
  float4* tw = gen_smem;
  float4* spw = tw + L::tw_len(ax);
  float2* spt = reinterpret_cast<float2*>(spw + rows * n);
  float2* bufs = spt + rows * n;
  float2* accs = bufs + rows * G * L::row_len(ax);
  float2* centre = accs + rows * G * n;
  float* sw = reinterpret_cast<float*>(centre + rows * n);
  float* srefs = sw + rows * n;
  const int b = a.probe0 + blockIdx.y;
  const int d = a.draw ? a.draw[b] : 0;
  const long long srow = (long long)d * a.n_slices + a.slice;
  const long long plane = (long long)a.ny * n;
  for (int i = threadIdx.x; i < L::tw_len(ax); i += blockDim.x) tw[i] = __ldg(L::twiddles(ax) + i);
  for (int i = threadIdx.x; i < a.K; i += blockDim.x) srefs[i] = __ldg(a.refs + srow * a.K + i);
  for (int i = threadIdx.x; i < (int)(sizeof(WpmSlice) / 4); i += blockDim.x)
    reinterpret_cast<int*>(&srec)[i] = __ldg(reinterpret_cast<const int*>(na.rec + srow) + i);
  for (int i = threadIdx.x; i < rows * G * n; i += blockDim.x) accs[i] = make_float2(0.f, 0.f);
  __syncthreads();
  const bool nodes = srec.nodes != 0;
  const int nf = srec.nf;
  const int row0 = blockIdx.x * rows, live_rows = min(rows, a.ny - row0);
  const long long at0 = (long long)row0 * n;
  const float* vs = a.V + (long long)d * a.v_draw_stride + (long long)a.slice * plane + at0;
  for (int i = threadIdx.x; i < live_rows * n; i += blockDim.x) {
    const WpmPixel px = wpm_pixel(__ldg(vs + i), srefs, a.K, a.ri_a, a.ri_inv_den, srec, na.spacing, na.kk);
    spw[i] = make_float4(px.pl.x, px.pl.y, px.pr.x, px.pr.y);
    spt[i] = make_float2(px.tl, px.tr);
    sw[i] = px.w;
  }
  __syncthreads();
  pdl_wait_then_release();

  // threads: group-major, then rows; what is left of the block only keeps the barriers
  const int g = threadIdx.x / (rows * T), in = threadIdx.x - g * rows * T;
  const int t = in % T;
  const bool mine = g < G && in / T < live_rows;
  const int rl = mine ? in / T : 0, slot = mine ? g * rows + rl : 0;
  const auto mem = L::row_mem(ax, bufs + min(g * rows + in / T, rows * G - 1) * L::row_len(ax));
  GenWpmBlend blend{nullptr, spw + rl * n, spt + rl * n, sw + rl * n, srec, accs + slot * n, centre + rl * n, 0, nodes};
  for (int k0 = 0; k0 < nf; k0 += G) {
    blend.k = k0 + g;
    blend.fk = a.fields + ((long long)b * a.K + blend.k) * plane + at0 + rl * n;
    L::pass(ax, tw, mem, t, mine && blend.k < nf, blend);
    __syncthreads();
  }
  float2* snap = a.snap ? a.snap + (long long)b * a.snap_bstride + at0 : nullptr;
  float2* wave = a.psi + (long long)b * plane + at0;
  const int shares = min(G, nf);
  for (int i = threadIdx.x; i < live_rows * n; i += blockDim.x) {
    float2 o = accs[i];
    for (int h = 1; h < shares; ++h) o = cadd(o, accs[h * rows * n + i]);
    if (nodes) {
      const float4 m = spw[i];
      const float2 y = centre[i];
      const float mx = m.x + m.z, my = m.y + m.w;
      o = make_float2(y.x + fmaf(y.x, mx, fmaf(-y.y, my, o.x)), y.y + fmaf(y.x, my, fmaf(y.y, mx, o.y)));
    }
    o = scale_hl(o, ga.scale);
    if (snap) __stcs(snap + i, o);
    if (a.last) __stcg(wave + i, o);
    centre[i] = o;
  }
  __syncthreads();
  GenWpmNext next{centre + rl * n, a.last ? a.dpbuf + (long long)b * a.dpbuf_bstride + at0 + rl * n : wave + rl * n};
  L::pass(ax, tw, mem, t, mine && g == 0, next);
}

// Blocks a column pass is split into along z, each with a share of the fields.
inline int gen_wpm_shares(const GenWpmColArgs& a, int blocks, int nb) {
  const WpmColArgs& c = a.n.c;
  const int z = c.dp_mode ? 1 : (long long)blocks * nb * 4 <= 592 ? 4 : (long long)blocks * nb * 2 <= 592 ? 2 : 1;
  return std::min(z, std::max(1, c.K));
}

// Shared memory of a row block.
inline size_t gen_wpm_row_bytes(const GenWpmRowArgs& a, int rows, int groups, int tw_len, int line_len) {
  const WpmRowArgs& r = a.n.r;
  return tw_len * sizeof(float4) + (size_t)rows * r.nx * (28 + 8 + 8 * groups) +
         (size_t)rows * groups * line_len * sizeof(float2) + r.K * sizeof(float);
}

// Bluestein axes (wap_bluestein.cu)
cudaError_t launch_blue_wcol(GenWpmColArgs& a, int nb, cudaStream_t st);
cudaError_t launch_blue_wrow(GenWpmRowArgs& a, int nb, cudaStream_t st);

}  // namespace wap
