// Mixed-radix line transforms for grid sides that are not powers of two.
//
// A length-n DFT runs as up to five Stockham stages of radices 2 .. 8 (n a
// product of such radices; sides with a prime above 7: wap_bluestein.cu).
// The radices are run-time values (any side, one kernel); larger ones (up to 16)
// halve the exchanges but not the time: their code, run once per block, and 200
// registers per thread made a 240 x 300 x 16 pass 91 us.
// A line belongs to T = n / (smallest radix) threads, one butterfly each per stage;
// stages exchange through two shared-memory buffers in turn (one barrier per stage).
// A pass over a line is a chain of DFTs with a pointwise product between them: the last stage of a transform and the first of the next have the
// same radix (every second transform takes the radices in reverse order), so the
// product happens in registers, and a pass of two S-stage transforms needs
// 2 S - 2 exchanges.  Inverse DFTs are forward ones of conjugates; the pointwise
// functions conjugate.
//
// All constants that repeat in every slice (butterfly constants, stage twiddles)
// are applied as float hi + lo parts, as in wap_fft.cuh.
#pragma once
#include "wap_passes.cuh"

namespace wap {

constexpr int kMixStages = 5;

// ---------------------------------------------------------------------------
// butterflies (forward sign), natural order in and out
// ---------------------------------------------------------------------------
// cos / sin of 2 pi j / P, j = 1 .. (P - 1) / 2, as float hi + lo
template <int P>
__device__ __forceinline__ Pair root_cos_half(int j) {
  if constexpr (P == 3) {
    if (j == 1) return {-5.000000000e-01f, 0.000000000e+00f};
  } else if constexpr (P == 5) {
    if (j == 1) return {3.090170026e-01f, -8.207602598e-09f};
    if (j == 2) return {-8.090170026e-01f, 8.207602598e-09f};
  } else if constexpr (P == 7) {
    if (j == 1) return {6.234897971e-01f, 4.743407445e-09f};
    if (j == 2) return {-2.225209326e-01f, -1.401115779e-09f};
    if (j == 3) return {-9.009688497e-01f, -1.824345297e-08f};
  }
  return {1.0f, 0.0f};
}
template <int P>
__device__ __forceinline__ Pair root_sin_half(int j) {
  if constexpr (P == 3) {
    if (j == 1) return {8.660253882e-01f, 1.554362505e-08f};
  } else if constexpr (P == 5) {
    if (j == 1) return {9.510565400e-01f, -2.371720598e-08f};
    if (j == 2) return {5.877852440e-01f, 8.304436250e-09f};
  } else if constexpr (P == 7) {
    if (j == 1) return {7.818315029e-01f, -2.044639835e-08f};
    if (j == 2) return {9.749279022e-01f, 9.960143821e-09f};
    if (j == 3) return {4.338837266e-01f, 1.252072579e-08f};
  }
  return {0.0f, 0.0f};
}
// cos / sin of 2 pi m / P (compile-time constants once the loops are unrolled)
template <int P>
__device__ __forceinline__ Pair root_cos(int m) {
  m %= P;
  return root_cos_half<P>(m <= P / 2 ? m : P - m);
}
template <int P>
__device__ __forceinline__ Pair root_sin(int m) {
  m %= P;
  const Pair s = root_sin_half<P>(m <= P / 2 ? m : P - m);
  return m <= P / 2 ? s : Pair{-s.hi, -s.lo};
}

// odd prime P: the cosine sums of x_j + x_{P-j} and the sine sums of x_j - x_{P-j}
template <int P>
__device__ __forceinline__ void mix_prime(float2 (&a)[P]) {
  constexpr int H = (P - 1) / 2;
  float2 t[H], s[H];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    t[j] = cadd(a[j + 1], a[P - 1 - j]);
    s[j] = csub(a[j + 1], a[P - 1 - j]);
  }
  const float2 a0 = a[0];
#pragma unroll
  for (int j = 0; j < H; ++j) a[0] = cadd(a[0], t[j]);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    float2 r = a0, i = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const Pair c = root_cos<P>((j + 1) * k), n = root_sin<P>((j + 1) * k);
      r = make_float2(fmaf(c.lo, t[j].x, r.x), fmaf(c.lo, t[j].y, r.y));
      i = make_float2(fmaf(n.lo, s[j].x, i.x), fmaf(n.lo, s[j].y, i.y));
    }
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const Pair c = root_cos<P>((j + 1) * k), n = root_sin<P>((j + 1) * k);
      r = make_float2(fmaf(c.hi, t[j].x, r.x), fmaf(c.hi, t[j].y, r.y));
      i = make_float2(fmaf(n.hi, s[j].x, i.x), fmaf(n.hi, s[j].y, i.y));
    }
    a[k] = make_float2(r.x + i.y, r.y - i.x);
    a[P - k] = make_float2(r.x - i.y, r.y + i.x);
  }
}

// 6 = 2 x 3 by the prime-factor index maps, no twiddles
__device__ __forceinline__ void mix_six(float2 (&a)[6]) {
  float2 e[3] = {a[0], a[2], a[4]}, o[3] = {a[3], a[5], a[1]};   // n = 3 i + 2 j mod 6
  mix_prime<3>(e);
  mix_prime<3>(o);
  // k = i mod 2, k = j mod 3
  a[0] = cadd(e[0], o[0]);
  a[3] = csub(e[0], o[0]);
  a[4] = cadd(e[1], o[1]);
  a[1] = csub(e[1], o[1]);
  a[2] = cadd(e[2], o[2]);
  a[5] = csub(e[2], o[2]);
}

template <int R>
__device__ __forceinline__ void mix_dft(float2 (&a)[R]) {
  if constexpr (R == 2 || R == 4 || R == 8) dft<R, false>(a);
  else if constexpr (R == 6) mix_six(a);
  else mix_prime<R>(a);
}

// ---------------------------------------------------------------------------
// one pass over a line
// ---------------------------------------------------------------------------
// Shared memory of a line: two buffers, position p at p * stride (rows: 1; lanes
// along the w columns of a tile: w).
struct MixMem {
  float2* buf;    // buffer 0 of this line
  int other;      // offset of buffer 1
  int stride;
};

// One stage, and with it the turn to the next transform where this stage ends one.
struct MixStep {
  int L, tw;           // span, offset of its twiddles
  float inv_L;
  const float2* src;   // buffer read, buffer written
  float2* dst;
  bool load, end, last;   // first stage of the pass; last of a transform; of the pass
};

template <int R, class Op>
__device__ __forceinline__ void mix_butterfly(const GenAxis& ax, const MixStep& st, const float4* tw, int stride, int b,
                                              Op& op) {
  const int nb = ax.m / R;
  float2 v[R];
  if (st.load) {
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = op.load(b + j * nb);
  } else {
    const float2* s = st.src + b * stride;
    const int d = nb * stride;
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = s[j * d];
  }
  int base = b * R;
  if (st.L > 1) {
    const int k = b - st.L * (int)(((float)b + 0.5f) * st.inv_L);   // b mod L (b < 2048: exact)
    const float4* w = tw + st.tw + k;
#pragma unroll
    for (int j = 1; j < R; ++j) v[j] = cmul_tw(v[j], w[(j - 1) * st.L]);
    base = (b - k) * R + k;
  }
  mix_dft<R>(v);
  int step = st.L;
  if (st.end) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int p = b + j * nb;
      if (st.last) op.store(p, v[j]);
      else v[j] = op.turn(p, v[j]);
    }
    if (st.last) return;
    mix_dft<R>(v);
    base = b * R;
    step = 1;
  }
  float2* o = st.dst + base * stride;
  const int d = step * stride;
#pragma unroll
  for (int j = 0; j < R; ++j) o[j * d] = v[j];
}

// `count` DFTs of the line (1 or 2): op.load(p) gives the input, op.turn(p, y) what
// the second DFT takes in place of the first's result y, op.store(p, y) takes the
// last one's result.  Every thread of the block calls it; `live` lines only do work.
template <class Op>
__device__ __forceinline__ void mix_pass(const GenAxis& ax, int count, const float4* tw, const MixMem& mem, int t,
                                         bool live, Op& op) {
  MixStep st;
  st.dst = mem.buf;
  st.src = mem.buf + mem.other;
  for (int g = 0; g < count; ++g) {
    int L = 1;
    st.tw = (g & 1) ? ax.tw_rev : 0;
    for (int s = 0; s < ax.stages; ++s) {
      const int R = ax.radix[(g & 1) ? ax.stages - 1 - s : s];
      st.L = L;
      st.inv_L = __fdividef(1.0f, (float)L);
      st.load = g == 0 && s == 0;
      st.end = s == ax.stages - 1;
      st.last = st.end && g == count - 1;
      if (s > 0 || g == 0) {   // (later transforms' first stage belongs to the turn)
        if (live) switch (R) {
#define WAP_MIX_CASE(r) case r: if (t * r < ax.m) mix_butterfly<r>(ax, st, tw, mem.stride, t, op); break;
          WAP_MIX_CASE(2) WAP_MIX_CASE(3) WAP_MIX_CASE(4) WAP_MIX_CASE(5) WAP_MIX_CASE(6) WAP_MIX_CASE(7)
          WAP_MIX_CASE(8)
#undef WAP_MIX_CASE
        }
        if (!st.last) __syncthreads();
        float2* done = st.dst;
        st.dst = const_cast<float2*>(st.src);
        st.src = done;
      }
      if (s > 0) st.tw += (R - 1) * L;
      L *= R;
    }
  }
}

}  // namespace wap
