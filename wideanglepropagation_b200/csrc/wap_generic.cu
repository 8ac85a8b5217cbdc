// Grids whose sides are not powers of two (any n in [17, 1024] per axis).
//
// The reference takes any n x m grid (get_frequencies, propagation.py:102-107,
// and jnp.fft.fft2 everywhere); its notebooks use e.g. gpts = 100
// (wpm/wpm_adaptive_comparison.ipynb).  Such a side's DFT runs on the mixed-radix
// lines of wap_mixed.cuh, a power-of-two side of such a grid too.
//
// Passes mirror the power-of-two ones (wap_passes.cuh): a row pass ([inverse row
// DFT, 1/(ny nx)] -> [snapshot] -> [* t] -> [row DFT]) and a column pass ([column
// DFT] -> [* H] -> [pattern] -> [inverse column DFT]); the WPM column pass forms
// the fields of a slice and its row pass blends them (wap_wpm_nodes.cuh has the
// method and the formulas of both).  All go out with programmatic dependent launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "wap_generic.cuh"
#include "wap_internal.h"

namespace wap {

__global__ void __launch_bounds__(2 * kGenThreads, 2) gen_row_kernel(const GenRowArgs a) {
  extern __shared__ float4 gen_smem[];
  const GenAxis& ax = a.ax;
  const int T = ax.threads, rows = a.rows;
  float4* tw = gen_smem;
  float2* bufs = reinterpret_cast<float2*>(tw + ax.tw_len);
  for (int i = threadIdx.x; i < ax.tw_len; i += blockDim.x) tw[i] = __ldg(ax.tw + i);
  const int rl = threadIdx.x / T, t = threadIdx.x - rl * T;
  const int row = blockIdx.x * rows + rl;
  const bool live = rl < rows && row < a.ny;
  const int b = a.probe0 + blockIdx.y;
  const bool first = a.flags & ROW_LOAD_SRC;
  if (first) pdl_wait_then_release();
  GenRowOp op = gen_row_op(a, b, row);
  const MixMem mem{bufs + min(rl, rows - 1) * ax.m, rows * ax.m, 1};
  if (a.fetch) {
    // the rows' transmission under the previous pass's tail
    float2* ts = bufs + 2 * rows * ax.m;
    const int row0 = blockIdx.x * rows, count = min(rows, a.ny - row0) * a.nx;
    const float2* src = op.trow + (row0 - row) * a.nx;
    for (int i = threadIdx.x; i < count; i += blockDim.x) ts[i] = __ldcg(src + i);
    op.trow = ts + rl * a.nx;
  }
  __syncthreads();
  if (!first) pdl_wait_then_release();
  mix_pass(ax, (a.flags & (ROW_IFFT | ROW_FFT)) == (ROW_IFFT | ROW_FFT) ? 2 : 1, tw, mem, t, live, op);
}

__global__ void __launch_bounds__(2 * kGenThreads, 2) gen_col_kernel(const GenColArgs a) {
  extern __shared__ float4 gen_smem[];
  const GenAxis& ax = a.ax;
  float4* tw = gen_smem;
  float2* bufs = reinterpret_cast<float2*>(tw + ax.tw_len);
  for (int i = threadIdx.x; i < ax.tw_len; i += blockDim.x) tw[i] = __ldg(ax.tw + i);
  const int w = a.w, c = threadIdx.x & (w - 1), t = threadIdx.x / w;
  const int col = blockIdx.x * w + c;
  const bool live = t < ax.threads && col < a.nx;
  const int b = a.probe0 + blockIdx.y;
  GenColOp op = gen_col_op(a, b, col);
  const MixMem mem{bufs + c, ax.m * w, w};
  if (a.fetch) {   // H, an input of the call, under the previous pass's tail
    float4* hs = reinterpret_cast<float4*>(bufs + 2 * ax.m * w);
    const int cols = min(w, a.nx - (int)blockIdx.x * w);
    for (int i = threadIdx.x; i < a.ny * w; i += blockDim.x) {
      const int r = i / w, k = i & (w - 1);
      if (k < cols) {
        const int o = r * a.nx + blockIdx.x * w + k;
        const float2 h = __ldg(a.H + o), l = a.H_lo ? __ldg(a.H_lo + o) : make_float2(0.f, 0.f);
        hs[i] = make_float4(h.x, h.y, l.x, l.y);
      }
    }
    op.hq = hs + c;
  }
  __syncthreads();
  pdl_wait_then_release();
  mix_pass(ax, 2, tw, mem, t, live, op);
}

// exp(i phi(V)) of every slice, any pixel count
__global__ void __launch_bounds__(256) gen_trans_table_kernel(const float* __restrict__ V, float2* __restrict__ ttab,
                                                              long long n, float a, float inv_den, float kphase) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    ttab[i] = transmission(__ldg(V + i), a, inv_den, kphase);
}

// ----------------------------------------------------------------------------
// launches
// ----------------------------------------------------------------------------
cudaError_t launch_gen_row(GenRowArgs& a, int nb, cudaStream_t st) {
  if (a.ax.blue) return launch_blue_row(a, nb, st);
  a.rows = gen_lines(a.ny, a.ax.threads, 64, std::max(1, 32 / a.ax.threads), kGenThreads, nb);
  a.fetch = a.tab_ready && (a.flags & ROW_TRANS_TAB) && gen_fetch(a.ax, (long long)a.ny * nb);
  const size_t smem =
      a.ax.tw_len * sizeof(float4) + (size_t)a.rows * (2 * a.ax.m + (a.fetch ? a.nx : 0)) * sizeof(float2);
  return launch_gen(gen_row_kernel, dim3((a.ny + a.rows - 1) / a.rows, nb), a.rows * a.ax.threads, smem, st, a);
}

static cudaError_t launch_gen_col(GenColArgs& a, int nb, cudaStream_t st) {
  if (a.ax.blue) return launch_blue_col(a, nb, st);
  a.w = gen_cols(a.ax, a.nx, nb);
  a.fetch = gen_fetch(a.ax, (long long)a.nx * nb);
  const size_t smem = a.ax.tw_len * sizeof(float4) +
                      (size_t)a.w * (2 * a.ax.m * sizeof(float2) + (a.fetch ? a.ny * sizeof(float4) : 0));
  return launch_gen(gen_col_kernel, dim3((a.nx + a.w - 1) / a.w, nb), a.w * a.ax.threads, smem, st, a);
}

// ----------------------------------------------------------------------------
// host: axis tables
// ----------------------------------------------------------------------------
bool generic_size_supported(int n) { return n >= 17 && n <= 1024; }

// The radices of a length-n transform: as few stages as possible, then the largest
// smallest radix (fewest threads per line); odd ones at both ends, where the stores
// of a stage of span 1 (stride R) then meet no bank conflicts.  false if a prime
// above 7 divides n or more than kMixStages are needed.
static bool plan_radices(int n, std::vector<int>* best) {
  best->clear();
  std::vector<int> cur;
  auto search = [&](auto&& self, int rest, int most) -> void {
    if (rest == 1) {
      if (best->empty() || cur.size() < best->size() || (cur.size() == best->size() && cur.back() > best->back()))
        *best = cur;
      return;
    }
    if ((int)cur.size() == kMixStages) return;
    for (int r = std::min(most, rest); r >= 2; --r) {
      if (rest % r) continue;
      cur.push_back(r);
      self(self, rest / r, r);
      cur.pop_back();
    }
  };
  search(search, n, 8);
  if (best->empty()) return false;
  std::stable_sort(best->begin(), best->end(), [](int a, int b) { return (a & 1) > (b & 1); });
  if (best->size() > 2 && ((*best)[1] & 1)) std::rotate(best->begin() + 1, best->begin() + 2, best->end());
  return true;
}

// DFT in float64 by recursion over the smallest factors (host; table set-up only)
static std::vector<std::complex<double>> host_dft(const std::vector<std::complex<double>>& x) {
  const int n = (int)x.size();
  if (n == 1) return x;
  int r = 2;
  while (n % r) ++r;
  const int q = n / r;
  std::vector<std::vector<std::complex<double>>> parts(r);
  for (int i = 0; i < r; ++i) {
    std::vector<std::complex<double>> sub(q);
    for (int j = 0; j < q; ++j) sub[j] = x[i + r * j];
    parts[i] = host_dft(sub);
  }
  std::vector<std::complex<double>> out(n);
  for (int k = 0; k < n; ++k)
    for (int i = 0; i < r; ++i) {
      const double ang = -2.0 * M_PI * (double)((long long)i * k % n) / (double)n;
      out[k] += parts[i][k % q] * std::complex<double>(std::cos(ang), std::sin(ang));
    }
  return out;
}

static float4 split(std::complex<double> z) {
  const float rh = (float)z.real(), ih = (float)z.imag();
  return make_float4(rh, ih, (float)(z.real() - (double)rh), (float)(z.imag() - (double)ih));
}

template <class T>
static int upload_vec(const T** dst, const std::vector<T>& v) {
  T* d = nullptr;
  cudaError_t e = cudaMalloc(&d, v.size() * sizeof(T));
  if (e == cudaSuccess) e = cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    return cuda_fail(e, "generic-axis table upload");
  }
  *dst = d;
  return WAP_OK;
}

// W_{L R}^{j k} of every stage after the first, [j - 1][k] within a stage
static void stage_twiddles(const std::vector<int>& radices, std::vector<float4>* tw) {
  int L = radices[0];
  for (size_t s = 1; s < radices.size(); ++s) {
    const int R = radices[s];
    const long long LR = (long long)L * R;
    for (int j = 1; j < R; ++j)
      for (int k = 0; k < L; ++k) {
        const double ang = -2.0 * M_PI * (double)((long long)j * k % LR) / (double)LR;
        tw->push_back(split({std::cos(ang), std::sin(ang)}));
      }
    L *= R;
  }
}

static int smooth_axis_tables(GenAxis* ax, const std::vector<int>& radices) {
  ax->stages = (int)radices.size();
  for (int s = 0; s < ax->stages; ++s) ax->radix[s] = radices[s];
  ax->threads = ax->m / *std::min_element(radices.begin(), radices.end());
  std::vector<float4> tw;
  stage_twiddles(radices, &tw);
  const std::vector<int> rev(radices.rbegin(), radices.rend());
  if (rev != radices) {
    ax->tw_rev = (int)tw.size();
    stage_twiddles(rev, &tw);
  }
  ax->tw_len = (int)tw.size();
  return upload_vec(&ax->tw, tw);
}

int generic_axis_create(GenAxis* ax, int n) {
  *ax = GenAxis{};
  ax->n = ax->m = n;
  std::vector<int> radices;
  if (plan_radices(n, &radices)) return smooth_axis_tables(ax, radices);
  // Bluestein through power-of-two lines in registers (wap_bluestein.cu)
  ax->blue = 1;
  ax->m = 64;
  while (ax->m < 2 * n - 1) ax->m <<= 1;
  std::vector<float4> tw = twiddle_table(ax->m, 8);
  ax->tw_rev = (int)tw.size();
  const std::vector<float4> tw16 = twiddle_table(ax->m, 16);
  tw.insert(tw.end(), tw16.begin(), tw16.end());
  ax->tw_len = (int)tw.size();
  int rc = upload_vec(&ax->tw, tw);
  if (rc) return rc;
  // chirp w_q = exp(-i pi q^2 / n) with q^2 reduced mod 2n (exact integers)
  const int m = ax->m;
  std::vector<float4> chirp(n);
  std::vector<std::complex<double>> bq(m, 0.0);
  for (int q = 0; q < n; ++q) {
    const long long r = ((long long)q * q) % (2LL * n);
    const double ang = M_PI * (double)r / (double)n;
    const std::complex<double> w(std::cos(ang), -std::sin(ang));
    chirp[q] = split(w);
    bq[q] = std::conj(w);
    if (q > 0) bq[m - q] = std::conj(w);
  }
  const std::vector<std::complex<double>> bf = host_dft(bq);
  std::vector<float4> hf(m);
  for (int i = 0; i < m; ++i) hf[i] = split(bf[i] / (double)m);
  if ((rc = upload_vec(&ax->chirp, chirp)) || (rc = upload_vec(&ax->bhat, hf))) return rc;
  return WAP_OK;
}

void generic_axis_free(GenAxis* ax) {
  cudaFree(const_cast<float4*>(ax->tw));
  cudaFree(const_cast<float4*>(ax->chirp));
  cudaFree(const_cast<float4*>(ax->bhat));
  *ax = GenAxis{};
}

// ----------------------------------------------------------------------------
// forward drivers
// ----------------------------------------------------------------------------
cudaError_t gen_trans_table(const float* V, float2* ttab, long long n, const RowArgs& r, cudaStream_t st) {
  gen_trans_table_kernel<<<(unsigned)std::min<long long>((n + 255) / 256, 148LL * 16), 256, 0, st>>>(
      V, ttab, n, r.ri_a, r.ri_inv_den, r.kphase);
  return cudaGetLastError();
}

int generic_fresnel_forward(wap_plan* p, const RowArgs& base, const ColArgs& cbase, int n_slices, int n_probes,
                            float2* stack, cudaStream_t st) {
  const long long plane = (long long)p->ny * p->nx;
  GenRowArgs r{};
  r.psi = base.psi;
  r.psi_bstride = plane;
  r.src = base.src;
  r.src_bstride = base.src_bstride;
  r.shifts = base.shifts;
  r.V = base.V;
  r.ttab = base.ttab;
  r.draw = base.draw;
  r.v_draw_stride = base.v_draw_stride;
  r.ax = p->gen_x;
  r.ny = p->ny;
  r.nx = p->nx;
  r.scale = inverse_scale(plane);
  r.ri_a = base.ri_a;
  r.ri_inv_den = base.ri_inv_den;
  r.kphase = base.kphase;
  GenColArgs c{};
  c.psi = base.psi;
  c.psi_bstride = plane;
  c.H = cbase.H;
  c.H_lo = cbase.H_lo;
  c.dp = cbase.dp;
  c.det = cbase.det;
  c.ax = p->gen_y;
  c.ny = p->ny;
  c.nx = p->nx;
  const int trans = base.ttab ? ROW_TRANS_TAB : ROW_TRANS;
  cudaError_t e;
  for (int b0 = 0; b0 < n_probes; b0 += 65535) {
    const int nb = std::min(65535, n_probes - b0);
    r.probe0 = c.probe0 = b0;
    for (int s = 0; s <= n_slices; ++s) {
      r.slice = s;
      r.tab_ready = s > 0;
      r.flags = (s == 0 ? ROW_LOAD_SRC : ROW_IFFT) | (s < n_slices ? (trans | ROW_FFT) : 0);
      r.snap = nullptr;
      if (stack && s >= 1) {
        r.snap = stack + (long long)(s - 1) * plane;
        r.snap_bstride = (long long)n_slices * plane;
      }
      if ((e = launch_gen_row(r, nb, st)) != cudaSuccess) return cuda_fail(e, "generic row pass");
      if (s == n_slices) break;
      c.flags = (s == n_slices - 1 && c.dp) ? COL_DP : 0;
      if ((e = launch_gen_col(c, nb, st)) != cudaSuccess) return cuda_fail(e, "generic column pass");
    }
  }
  return WAP_OK;
}

}  // namespace wap
