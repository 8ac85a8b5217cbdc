// WPM on grids whose sides are not powers of two: the mixed-radix kernels and the
// forward driver (wap_generic_wpm.cuh has the passes).
#include <cuda_runtime.h>

#include <algorithm>

#include "wap_generic_wpm.cuh"
#include "wap_internal.h"

namespace wap {

struct MixLine {
  static constexpr int kCol = 2 * kGenThreads, kColBlocks = 2;
  static __device__ __forceinline__ int threads(const GenAxis& ax) { return ax.threads; }
  static __device__ __forceinline__ int tw_len(const GenAxis& ax) { return ax.tw_len; }
  static __device__ __forceinline__ const float4* twiddles(const GenAxis& ax) { return ax.tw; }
  static __device__ __forceinline__ int col_len(const GenAxis& ax) { return 2 * ax.m; }
  static __device__ __forceinline__ int row_len(const GenAxis& ax) { return 2 * ax.m; }
  static __device__ __forceinline__ MixMem col_mem(const GenAxis& ax, float2* bufs, int w, int c) {
    return {bufs + c, ax.m * w, w};
  }
  static __device__ __forceinline__ MixMem row_mem(const GenAxis& ax, float2* buf) { return {buf, ax.m, 1}; }
  template <class Op>
  static __device__ __forceinline__ void pass(const GenAxis& ax, const float4* tw, const MixMem& mem, int t, bool live,
                                              Op& op) {
    mix_pass(ax, 1, tw, mem, t, live, op);
  }
};

static cudaError_t launch_gen_wcol(GenWpmColArgs& a, int nb, cudaStream_t st) {
  if (a.ax.blue) return launch_blue_wcol(a, nb, st);
  const WpmColArgs& c = a.n.c;
  a.w = gen_cols(a.ax, c.nx, nb);
  const size_t smem = a.ax.tw_len * sizeof(float4) + 3 * (size_t)a.ax.m * a.w * sizeof(float2);
  const int blocks = (c.nx + a.w - 1) / a.w;
  return launch_gen(a.refs ? gen_wpm_col_kernel<MixLine, true> : gen_wpm_col_kernel<MixLine, false>,
                    dim3(blocks, nb, gen_wpm_shares(a, blocks, nb)), a.w * a.ax.threads, smem, st, a);
}

static cudaError_t launch_gen_wrow(GenWpmRowArgs& a, int nb, cudaStream_t st) {
  if (a.ax.blue) return launch_blue_wrow(a, nb, st);
  const WpmRowArgs& r = a.n.r;
  const int T = a.ax.threads;
  auto bytes = [&](int rows, int groups) { return gen_wpm_row_bytes(a, rows, groups, a.ax.tw_len, 2 * a.ax.m); };
  a.groups = std::max(1, std::min({4, 2 * kGenThreads / T, r.K}));
  a.rows = gen_lines(r.ny, T * a.groups, 64, std::max(1, 32 / (T * a.groups)), 2 * kGenThreads, nb);
  while (a.rows > 1 && bytes(a.rows, a.groups) > kGenSmem / 2) a.rows = (a.rows + 1) / 2;
  while (a.groups > 1 && bytes(a.rows, a.groups) > kGenSmem) --a.groups;
  return launch_gen(gen_wpm_row_kernel<MixLine>, dim3((r.ny + a.rows - 1) / a.rows, nb), a.rows * a.groups * T,
                    bytes(a.rows, a.groups), st, a);
}

int generic_wpm_forward(const wap_plan* p, const WpmColArgs& cbase, const WpmRowArgs& wbase,
                        const WpmNodeScalars& nodes, double power, const float2* psi0, long long psi0_stride,
                        const int32_t* positions, int n_slices, int n_probes, float* dp, float2* stack,
                        cudaStream_t st) {
  const long long plane = (long long)p->ny * p->nx;
  cudaError_t e;
  GenRowArgs r{};
  r.psi = wbase.psi;
  r.psi_bstride = plane;
  r.src = psi0;
  r.src_bstride = psi0_stride;
  r.shifts = positions;
  r.ax = p->gen_x;
  r.ny = p->ny;
  r.nx = p->nx;
  r.flags = ROW_LOAD_SRC | ROW_FFT;
  GenWpmColArgs c{wpm_node_col_args(p, cbase, nodes), p->gen_y, 0, !nodes.nodes};
  GenWpmRowArgs w{wpm_node_row_args(p, wbase, nodes, power), p->gen_x, inverse_scale(plane), 0, 0};
  for (int b0 = 0; b0 < n_probes; b0 += 65535) {
    const int nb = std::min(65535, n_probes - b0);
    r.probe0 = c.n.c.probe0 = w.n.r.probe0 = b0;
    if ((e = launch_gen_row(r, nb, st)) != cudaSuccess) return cuda_fail(e, "generic wpm row pass");
    for (int s = 0; s < n_slices; ++s) {
      c.n.c.slice = w.n.r.slice = s;
      c.n.c.dp_mode = 0;
      if ((e = launch_gen_wcol(c, nb, st)) != cudaSuccess) return cuda_fail(e, "generic wpm column pass");
      w.n.r.last = (s == n_slices - 1);
      w.n.r.snap = stack ? stack + (long long)s * plane : nullptr;
      if ((e = launch_gen_wrow(w, nb, st)) != cudaSuccess) return cuda_fail(e, "generic wpm row pass");
    }
    if (dp) {
      GenWpmColArgs d = c;
      d.n.c.psi = p->dpbuf;
      d.n.c.dp = dp;
      d.n.c.dp_mode = 1;
      if ((e = launch_gen_wcol(d, nb, st)) != cudaSuccess) return cuda_fail(e, "generic wpm pattern pass");
    }
  }
  return WAP_OK;
}

}  // namespace wap
