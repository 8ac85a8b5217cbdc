// Passes along sides with a prime factor above 7: Bluestein's chirp convolution,
//
//   X_k = w_k sum_j (x_j w_j) conj(w_{k-j}),   w_q = exp(-i pi q^2 / n),
//
// through the power-of-two FFT core (wap_fft.cuh) of length m >= 2 n - 1, a line's
// m-point vector in registers.  The pointwise functions are those of the
// mixed-radix passes (wap_generic.cuh, wap_generic_wpm.cuh).  Against the same
// convolution on mixed-radix lines of a shorter smooth length: 455^2 x 14 slices
// 0.44 ms here, 0.82 there; 1021^2 x 10 1.05, 1.97; WPM, 101^2 x 20, K = 8, 32 probes
// 1.41, 4.57, one probe 0.35, 0.85.
#include <cuda_runtime.h>

#include <algorithm>

#include "wap_generic.cuh"
#include "wap_generic_wpm.cuh"
#include "wap_internal.h"

namespace wap {

// `count` length-n DFTs of the line held as x[t + T e] (positions >= n are zero on
// input and ignored on output), the pointwise functions between and around them
template <int M, int E, class X, class Op>
__device__ __forceinline__ void blue_pass(const GenAxis& ax, int count, const float4* tw, const X& xs, int t, bool live,
                                          Op& op) {
  constexpr int T = M / E;
  float2 v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int p = t + T * e;
    v[e] = live && p < ax.n ? op.load(p) : make_float2(0.f, 0.f);
  }
  for (int c = 1; c <= count; ++c) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (t + T * e < ax.n) v[e] = cmul_tw(v[e], __ldg(ax.chirp + t + T * e));
    fft<M, E, false>(v, t, xs, tw);
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cmul_tw(v[e], __ldg(ax.bhat + t + T * e));
    fft<M, E, true>(v, t, xs, tw);
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int p = t + T * e;
      if (live && p < ax.n) {
        v[e] = cmul_tw(v[e], __ldg(ax.chirp + p));
        if (c < count) v[e] = op.turn(p, v[e]);
        else op.store(p, v[e]);
      } else {
        v[e] = make_float2(0.f, 0.f);
      }
    }
  }
}

template <int M, int E>
__global__ void __launch_bounds__(kRowThreads) blue_row_kernel(const GenRowArgs a) {
  constexpr int T = M / E;
  constexpr int PADN = RowExchange<true>::padded(M);
  extern __shared__ float4 blue_smem[];
  float4* tw = blue_smem;
  float2* xbuf = reinterpret_cast<float2*>(tw + FFTPlan<M, E>::TW_SIZE);
  const float4* src = a.ax.tw + (E == 16 ? a.ax.tw_rev : 0);
  for (int i = threadIdx.x; i < FFTPlan<M, E>::TW_SIZE; i += blockDim.x) tw[i] = __ldg(src + i);
  const int rl = threadIdx.x / T, t = threadIdx.x - rl * T;
  const int row = blockIdx.x * a.rows + rl;
  const bool live = row < a.ny;
  const bool first = a.flags & ROW_LOAD_SRC;
  if (first) pdl_wait_then_release();
  GenRowOp op = gen_row_op(a, a.probe0 + blockIdx.y, live ? row : 0);
  const RowExchange<(T <= 32)> xs{xbuf + rl * PADN};
  __syncthreads();
  if (!first) pdl_wait_then_release();
  blue_pass<M, E>(a.ax, (a.flags & (ROW_IFFT | ROW_FFT)) == (ROW_IFFT | ROW_FFT) ? 2 : 1, tw, xs, t, live, op);
}

template <int M, int E>
__global__ void __launch_bounds__(kColThreads) blue_col_kernel(const GenColArgs a) {
  extern __shared__ float4 blue_smem[];
  float4* tw = blue_smem;
  float2* tile = reinterpret_cast<float2*>(tw + FFTPlan<M, E>::TW_SIZE);
  const float4* src = a.ax.tw + (E == 16 ? a.ax.tw_rev : 0);
  for (int i = threadIdx.x; i < FFTPlan<M, E>::TW_SIZE; i += blockDim.x) tw[i] = __ldg(src + i);
  const int c = threadIdx.x & (a.w - 1), t = threadIdx.x / a.w;
  const int col = blockIdx.x * a.w + c;
  const bool live = col < a.nx;
  GenColOp op = gen_col_op(a, a.probe0 + blockIdx.y, live ? col : 0);
  const ColExchange<> xs{tile, a.w, c};
  __syncthreads();
  pdl_wait_then_release();
  blue_pass<M, E>(a.ax, 2, tw, xs, t, live, op);
}

// the wide-angle passes (wap_generic_wpm.cuh) on these lines.  A row block is groups x
// rows x T threads, all of them: the rows of a warp share its exchanges.
template <int M, int E>
struct BlueLine {
  static constexpr int T = M / E, kCol = kColThreads;
  static constexpr int kColBlocks = E == 8 ? 1 : 0;   // (asking for one block doubles the spills of 16 elements)
  using Row = RowExchange<(T <= 32)>;
  static __device__ __forceinline__ int threads(const GenAxis&) { return T; }
  static __device__ __forceinline__ int tw_len(const GenAxis&) { return FFTPlan<M, E>::TW_SIZE; }
  static __device__ __forceinline__ const float4* twiddles(const GenAxis& ax) {
    return ax.tw + (E == 16 ? ax.tw_rev : 0);
  }
  static __device__ __forceinline__ int col_len(const GenAxis&) { return M; }
  static __device__ __forceinline__ int row_len(const GenAxis&) { return Row::padded(M); }
  static __device__ __forceinline__ ColExchange<> col_mem(const GenAxis&, float2* bufs, int w, int c) {
    return {bufs, w, c};
  }
  static __device__ __forceinline__ Row row_mem(const GenAxis&, float2* buf) { return {buf}; }
  template <class X, class Op>
  static __device__ __forceinline__ void pass(const GenAxis& ax, const float4* tw, const X& xs, int t, bool live,
                                              Op& op) {
    blue_pass<M, E>(ax, 1, tw, xs, t, live, op);
  }
};

template <int M, int E>
static cudaError_t launch_row_t(GenRowArgs& a, int nb, cudaStream_t st) {
  constexpr int T = M / E;
  // rows of a warp share its exchanges: whole warps of rows
  a.rows = std::max(1, kRowThreads / T);
  while (a.rows > 1 && a.rows * T > 32 && (long long)((a.ny + a.rows - 1) / a.rows) * nb < 296) a.rows >>= 1;
  const size_t smem = FFTPlan<M, E>::TW_SIZE * sizeof(float4) + (size_t)a.rows * RowExchange<true>::padded(M) * 8;
  return launch_gen(blue_row_kernel<M, E>, dim3((a.ny + a.rows - 1) / a.rows, nb), a.rows * T, smem, st, a);
}

template <int M, int E>
static cudaError_t launch_col_t(GenColArgs& a, int nb, cudaStream_t st) {
  constexpr int T = M / E;
  a.w = std::max(1, std::min(16, kColThreads / T));
  while (a.w > 4 && a.w * T > 32 && (long long)((a.nx + a.w - 1) / a.w) * nb < 296) a.w >>= 1;
  const size_t smem = FFTPlan<M, E>::TW_SIZE * sizeof(float4) + (size_t)M * a.w * sizeof(float2);
  return launch_gen(blue_col_kernel<M, E>, dim3((a.nx + a.w - 1) / a.w, nb), a.w * T, smem, st, a);
}

template <int M, int E>
static cudaError_t launch_wcol_t(GenWpmColArgs& a, int nb, cudaStream_t st) {
  constexpr int T = M / E;
  const int nx = a.n.c.nx;
  a.w = std::max(1, std::min(16, kColThreads / T));
  while (a.w > 4 && a.w * T > 32 && (long long)((nx + a.w - 1) / a.w) * nb < 296) a.w >>= 1;
  const size_t smem = FFTPlan<M, E>::TW_SIZE * sizeof(float4) + (size_t)(M + a.ax.n) * a.w * sizeof(float2);
  const int blocks = (nx + a.w - 1) / a.w;
  return launch_gen(a.refs ? gen_wpm_col_kernel<BlueLine<M, E>, true> : gen_wpm_col_kernel<BlueLine<M, E>, false>,
                    dim3(blocks, nb, gen_wpm_shares(a, blocks, nb)), a.w * T, smem, st, a);
}

template <int M, int E>
static cudaError_t launch_wrow_t(GenWpmRowArgs& a, int nb, cudaStream_t st) {
  constexpr int T = M / E;
  const int ny = a.n.r.ny;
  auto bytes = [&] {
    return gen_wpm_row_bytes(a, a.rows, a.groups, FFTPlan<M, E>::TW_SIZE, RowExchange<true>::padded(M));
  };
  // several groups of threads per row while the rows alone leave the chip idle
  a.groups = 1;
  if ((long long)ny * nb * T <= 148LL * 256)
    while (a.groups < 4 && 2 * a.groups * T <= 2 * kGenThreads && 2 * a.groups <= a.n.r.K) a.groups *= 2;
  a.rows = std::max(1, (a.groups > 1 ? 2 * kGenThreads : kGenThreads) / (T * a.groups));
  while (a.rows > 1 && a.rows * a.groups * T > 32 &&
         (bytes() > kGenSmem / 2 || (long long)((ny + a.rows - 1) / a.rows) * nb < 296))
    a.rows >>= 1;
  return launch_gen(gen_wpm_row_kernel<BlueLine<M, E>>, dim3((ny + a.rows - 1) / a.rows, nb), a.rows * a.groups * T,
                    bytes(), st, a);
}

// 16 elements per thread (fewer exchanges) where the lines fill the chip, 8 (shorter
// chains, more warps) below
static bool blue_wide(int m, long long lines) { return lines * (m / 16) >= 148LL * 512; }

#define WAP_BLUE_SIZES(X) X(64) X(128) X(256) X(512) X(1024) X(2048)
#define WAP_BLUE_ROW(M) \
  case M: return blue_wide(M, (long long)a.ny * nb) ? launch_row_t<M, 16>(a, nb, st) : launch_row_t<M, 8>(a, nb, st);
#define WAP_BLUE_COL(M) \
  case M: return blue_wide(M, (long long)a.nx * nb) ? launch_col_t<M, 16>(a, nb, st) : launch_col_t<M, 8>(a, nb, st);

// (the wide-angle column pass holds more per element: 16 only where 8 would leave two
// columns per block.  32 probes, K = 2: 202^2 x 10 1.95 ms with 8, 2.02 with 16; 509^2
// x 4 5.55, 5.26; 1009^2 x 2 14.6, 12.9)
#define WAP_BLUE_WCOL(M)                                                                  \
  case M:                                                                                 \
    if (M >= 1024 && blue_wide(M, (long long)a.n.c.nx * nb))                              \
      return launch_wcol_t<M, (M >= 1024 ? 16 : 8)>(a, nb, st);                           \
    return launch_wcol_t<M, 8>(a, nb, st);
#define WAP_BLUE_WROW(M) \
  case M: return blue_wide(M, (long long)a.n.r.ny * nb) ? launch_wrow_t<M, 16>(a, nb, st) : launch_wrow_t<M, 8>(a, nb, st);

cudaError_t launch_blue_row(GenRowArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_ROW) default: return cudaErrorInvalidValue; }
}
cudaError_t launch_blue_col(GenColArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_COL) default: return cudaErrorInvalidValue; }
}

cudaError_t launch_blue_wcol(GenWpmColArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_WCOL) default: return cudaErrorInvalidValue; }
}
cudaError_t launch_blue_wrow(GenWpmRowArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_WROW) default: return cudaErrorInvalidValue; }
}

}  // namespace wap
