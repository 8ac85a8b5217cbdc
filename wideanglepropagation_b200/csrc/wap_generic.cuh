// What the translation units of the grids that are not powers of two share
// (wap_generic.cu: Fresnel / AS passes and the axis tables; wap_bluestein.cu: those
// passes along sides with a large prime factor; wap_generic_wpm.cu: WPM).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "wap_internal.h"
#include "wap_mixed.cuh"

namespace wap {

__device__ __forceinline__ int pmod(int a, int n) {
  const int r = a % n;
  return r < 0 ? r + n : r;
}

// fftshift position of index k on an n-point axis (numpy roll by n // 2)
__device__ __forceinline__ int shifted(int k, int n) {
  const int s = k + (n >> 1);
  return s >= n ? s - n : s;
}

// y s with s = hi + lo: 1/(ny nx) is no power of two here, and its rounding would
// scale the wave alike in every slice
__device__ __forceinline__ float2 scale_hl(float2 y, float2 s) {
  return make_float2(fmaf(y.x, s.x, y.x * s.y), fmaf(y.y, s.x, y.y * s.y));
}

constexpr int kGenThreads = 256;

struct GenRowArgs {
  float2* psi;
  long long psi_bstride;
  const float2* src;          // ROW_LOAD_SRC: initial wave(s)
  long long src_bstride;
  const int* shifts;          // (B, 2) probe centres or null
  const float* V;             // ROW_TRANS: (draws, n_slices, ny, nx) volts
  const float2* ttab;         // ROW_TRANS_TAB: exp(i phi(V)) laid out like V
  const int* draw;
  long long v_draw_stride;
  float2* snap;               // spatial wave entering `slice`, or null
  long long snap_bstride;
  GenAxis ax;                 // along x
  int ny, nx, slice, flags, probe0;
  int rows;                   // per block
  int tab_ready;              // ttab was complete two launches ago
  int fetch;                  // its rows go to shared memory before the wait
  float2 scale;               // after the inverse row DFT, hi + lo
  float ri_a, ri_inv_den, kphase;
};

// exp(i phi(V)) without a table (tables above 1 GiB), out of line: the row kernel
// holds one copy of its pointwise functions per radix
static __device__ __noinline__ float2 gen_transmission(float v, float a, float inv_den, float kphase) {
  return transmission(v, a, inv_den, kphase);
}

// the pointwise functions of a row pass on one row
struct GenRowOp {
  const GenRowArgs& a;
  float2* prow;
  const float2* srow;
  float2* snap;
  const float* vrow;
  const float2* trow;         // the row's table, or its copy in shared memory
  int sx, f;
  // the spatial value of the transformed line (or of the source) -> the value to transform
  __device__ __forceinline__ float2 slice_value(int p, float2 y) const {
    if (snap) __stcs(snap + p, y);
    if (f & ROW_TRANS_TAB) y = cmul(y, trow[p]);
    else if (f & ROW_TRANS) y = cmul(y, gen_transmission(__ldg(vrow + p), a.ri_a, a.ri_inv_den, a.kphase));
    return y;
  }
  __device__ __forceinline__ float2 load(int p) const {
    if (f & ROW_LOAD_SRC) {
      int x = p - sx;
      x += x < 0 ? a.nx : 0;
      return slice_value(p, __ldg(srow + x));
    }
    const float2 v = __ldcg(prow + p);
    return (f & ROW_IFFT) ? cconj(v) : v;
  }
  __device__ __forceinline__ float2 turn(int p, float2 y) const { return slice_value(p, scale_hl(cconj(y), a.scale)); }
  __device__ __forceinline__ void store(int p, float2 y) const {
    if (!(f & ROW_FFT)) {   // the inverse transform ends the pass: the spatial wave
      y = scale_hl(cconj(y), a.scale);
      if (snap) __stcs(snap + p, y);
    }
    __stcg(prow + p, y);
  }
};

// Reads the call's positions and draw indices.  The kernel before the first pass of a
// call (ROW_LOAD_SRC) may be the one that writes them, and its writes are visible only
// after the dependent-launch wait, so that pass waits before it comes here; later
// passes come here ahead of their wait, two launches after whatever wrote them.
__device__ __forceinline__ GenRowOp gen_row_op(const GenRowArgs& a, int b, int row) {
  GenRowOp op{a};
  op.f = a.flags;
  op.sx = 0;
  op.prow = a.psi + (long long)b * a.psi_bstride + row * a.nx;
  op.snap = a.snap ? a.snap + (long long)b * a.snap_bstride + row * a.nx : nullptr;
  const int plane = a.ny * a.nx;
  const int d = a.draw ? a.draw[b] : 0;
  const long long vat = (long long)d * a.v_draw_stride + (long long)a.slice * plane + row * a.nx;
  op.vrow = a.V + vat;
  op.trow = a.ttab + vat;
  int srow = row;
  if ((a.flags & ROW_LOAD_SRC) && a.shifts) {   // move_probe (propagation.py:263-276)
    srow = pmod(row - pmod(a.shifts[2 * b] - (a.ny >> 1), a.ny), a.ny);
    op.sx = pmod(a.shifts[2 * b + 1] - (a.nx >> 1), a.nx);
  }
  op.srow = a.src + (long long)b * a.src_bstride + srow * a.nx;
  return op;
}

// |y|^2 at (k_y = p, this column) of the fftshifted pattern's window
__device__ __forceinline__ void gen_pattern(float* dp, const Detector& det, int drx, int p, int ny, float2 y) {
  const int ry = shifted(p, ny) - det.y0;
  if ((unsigned)drx < (unsigned)det.nx && (unsigned)ry < (unsigned)det.ny)
    __stcs(dp + ry * det.nx + drx, fmaf(y.x, y.x, y.y * y.y));
}

struct GenColArgs {
  float2* psi;
  long long psi_bstride;
  const float2* H;            // (ny, nx)
  const float2* H_lo;
  float* dp;                  // COL_DP: (B, det window)
  Detector det;
  GenAxis ax;                 // along y
  int ny, nx, w, flags, probe0;   // w: columns per block
  int fetch;                  // H goes to shared memory before the wait
};

struct GenColOp {
  const GenColArgs& a;
  float2* pcol;
  const float2* hcol;
  const float2* lcol;
  const float4* hq;           // this column's (hi, lo) in shared memory, stride w, or null
  float* dp;
  int drx;
  __device__ __forceinline__ float2 load(int p) const { return __ldcg(pcol + p * a.nx); }
  __device__ __forceinline__ float2 turn(int p, float2 y) const {
    if (hq) {
      y = cmul_tw(y, hq[p * a.w]);
    } else {
      const int o = p * a.nx;
      y = lcol ? cmul_hl(y, __ldg(hcol + o), __ldg(lcol + o)) : cmul(y, __ldg(hcol + o));
    }
    if (dp) gen_pattern(dp, a.det, drx, p, a.ny, y);
    return cconj(y);
  }
  __device__ __forceinline__ void store(int p, float2 y) const { __stcg(pcol + p * a.nx, cconj(y)); }
};

__device__ __forceinline__ GenColOp gen_col_op(const GenColArgs& a, int b, int col) {
  GenColOp op{a};
  op.pcol = a.psi + (long long)b * a.psi_bstride + col;
  op.hcol = a.H + col;
  op.lcol = a.H_lo ? a.H_lo + col : nullptr;
  op.hq = nullptr;
  op.dp = (a.flags & COL_DP) ? a.dp + (long long)b * a.det.plane() : nullptr;
  op.drx = shifted(col, a.nx) - a.det.x0;
  return op;
}

// ----------------------------------------------------------------------------
// launches
// ----------------------------------------------------------------------------
constexpr size_t kGenSmem = 200 * 1024;

template <class K, class A>
inline cudaError_t launch_gen(K kern, dim3 grid, int threads, size_t smem, cudaStream_t st, const A& a) {
  cudaError_t e;
  if (beyond_default_smem(smem) &&
      (e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess)
    return e;
  count_launch();
  return launch_pdl(kern, grid, (threads + 31) & ~31, smem, st, a);
}

// Lines per block: up to `most` of `threads` threads each, fewer (down to `least`)
// while the grid has under two blocks per SM: a pass of one probe on 100^2 is 1000
// threads in all, and its time the chain of one line.
inline int gen_lines(int lines, int threads, int most, int least, int limit, int nb) {
  int per = std::max(1, std::min(most, limit / threads));
  while (per > least && (long long)((lines + per - 1) / per) * nb < 296) per = (per + 1) / 2;
  return std::min(per, lines);
}

// columns per block (a power of two): up to 16, down to 4 (32-byte row segments)
inline int gen_cols(const GenAxis& ax, int nx, int nb) {
  int w = 16;
  while (w > 1 && w * ax.threads > kGenThreads) w >>= 1;
  while (w > 4 && (long long)((nx + w - 1) / w) * nb < 296) w >>= 1;
  return w;
}

inline float2 inverse_scale(long long plane) {
  const double s = 1.0 / (double)plane;
  return make_float2((float)s, (float)(s - (double)(float)s));
}

// Whether a pass of `lines` lines is short of threads (under half the chip's): then its
// tables are copied to shared memory before the wait, off the chain of the pass
// (100^2, 100 slices: 1.23 -> 0.98 ms); a fuller pass hides their latency and the
// copy costs (1000^2, 20 slices: 1.24 -> 1.47 ms).
inline bool gen_fetch(const GenAxis& ax, long long lines) { return lines * ax.threads <= 148LL * 1024; }

cudaError_t launch_gen_row(GenRowArgs& a, int nb, cudaStream_t st);
// Bluestein axes of Fresnel / AS plans (wap_bluestein.cu)
cudaError_t launch_blue_row(GenRowArgs& a, int nb, cudaStream_t st);
cudaError_t launch_blue_col(GenColArgs& a, int nb, cudaStream_t st);

}  // namespace wap
