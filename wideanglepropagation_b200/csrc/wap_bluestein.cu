// Fresnel / AS passes along sides with a prime factor above 7: Bluestein's chirp
// convolution,
//
//   X_k = w_k sum_j (x_j w_j) conj(w_{k-j}),   w_q = exp(-i pi q^2 / n),
//
// through the power-of-two FFT core (wap_fft.cuh) of length m >= 2 n - 1, a line's
// m-point vector in registers.  The pointwise functions are those of the
// mixed-radix passes (wap_generic.cuh).  Against the same convolution on
// mixed-radix lines of a shorter smooth length (which the WPM passes use, where
// the transforms are a smaller share): 455^2 x 14 slices 0.82 ms there, 1021^2 x 10
// 1.97 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "wap_generic.cuh"
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
  constexpr int T = M / E;
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

// 16 elements per thread (fewer exchanges) where the lines fill the chip, 8 (shorter
// chains, more warps) below
static bool blue_wide(int m, long long lines) { return lines * (m / 16) >= 148LL * 512; }

#define WAP_BLUE_SIZES(X) X(64) X(128) X(256) X(512) X(1024) X(2048)
#define WAP_BLUE_ROW(M) \
  case M: return blue_wide(M, (long long)a.ny * nb) ? launch_row_t<M, 16>(a, nb, st) : launch_row_t<M, 8>(a, nb, st);
#define WAP_BLUE_COL(M) \
  case M: return blue_wide(M, (long long)a.nx * nb) ? launch_col_t<M, 16>(a, nb, st) : launch_col_t<M, 8>(a, nb, st);

cudaError_t launch_blue_row(GenRowArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_ROW) default: return cudaErrorInvalidValue; }
}
cudaError_t launch_blue_col(GenColArgs& a, int nb, cudaStream_t st) {
  switch (a.ax.m) { WAP_BLUE_SIZES(WAP_BLUE_COL) default: return cudaErrorInvalidValue; }
}

}  // namespace wap
