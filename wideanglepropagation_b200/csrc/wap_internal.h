// Internal declarations shared by the libwap.so translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "../../include/wap.h"

namespace wap {
// Detector window of a diffraction pattern: rows y0 .. y0+ny-1 and columns
// x0 .. x0+nx-1 of the fftshifted |fft2(psi)|^2 - the centre crop of
// downsample_to_max_angle (propagation.py:424-439).  A plan keeps ny == 0 for
// "the whole grid"; kernels always receive a resolved window.
struct Detector {
  int y0 = 0, x0 = 0, ny = 0, nx = 0;
  __host__ __device__ Detector resolved(int gy, int gx) const { return ny == 0 ? Detector{0, 0, gy, gx} : *this; }
  // pixels of one probe's pattern
  __host__ __device__ long long plane() const { return (long long)ny * nx; }
};

struct WpmSlice;   // a slice's WPM record (wap_wpm_nodes.cuh)

// One axis of a grid that is not a power of two: a length-n DFT by stages of radices
// 2 .. 8 (wap_mixed.cuh; m = n), or, with blue, as Bluestein's chirp convolution
// through transforms of a power of two m >= 2n - 1 (wap_bluestein.cu).  Device
// pointers; tables of float64 values stored as float hi + lo parts.
struct GenAxis {
  int n = 0, m = 0, blue = 0, stages = 0;
  int radix[5] = {0, 0, 0, 0, 0};
  int threads = 0;                  // per line: n / smallest radix
  int tw_rev = 0, tw_len = 0;       // offset of the second table, entries of both
  const float4* tw = nullptr;       // stage twiddles, radices in order, then in reverse order
                                    // (blue: the m-point tables of 8, then of 16 elements per thread)
  const float4* chirp = nullptr;    // (n) w_p = exp(-i pi p^2 / n)
  const float4* bhat = nullptr;     // (m) fft_m(b) / m, b_q = conj(w_q) on the circular index range
};
}  // namespace wap

struct wap_plan {
  int device = 0;
  int ny = 0, nx = 0, max_batch = 0, op = 0, n_bins = 0;
  int row_e = 16, col_e = 16, col_w = 16;   // FFT launch shape (autotuned)
  bool exact_shape = false;                 // set by the caller: launched as it is (else row_chunks, col_chunks)
  float4* tw_row = nullptr;                 // twiddles for nx / row_e (hi, lo)
  float4* tw_col = nullptr;                 // twiddles for ny / col_e (hi, lo)
  float4* tw_row8 = nullptr;                // the same for 8 elements per thread (medium passes),
  float4* tw_col8 = nullptr;                // where row_e / col_e are 16 and the side allows it
  // WPM workspace
  float2* fields = nullptr;                 // (max_batch, n_bins, ny, nx)
  float2* dpbuf = nullptr;                  // (max_batch, ny, nx)
  float2* blend = nullptr;                  // (max_batch, ny, nx) WPM bin-split blend
  float2* hvac = nullptr;                   // (ny, nx) hi part
  float2* hvac_lo = nullptr;                // (ny, nx) lo part
  float* ky2 = nullptr;
  float* kx2 = nullptr;
  float* q = nullptr;                       // (ny, nx) k0^2 - k_perp^2
  double hvac_key[4] = {0, 0, 0, 0};        // (dy, dx, dz, energy) of hvac
  float* refs = nullptr;                    // (draws, n_slices, n_bins)
  size_t refs_cap = 0;
  wap::WpmSlice* slices = nullptr;          // (draws, n_slices) interpolation records
  size_t slices_cap = 0;
  float4* wn_tw_row = nullptr;              // (nx, 8) and (ny, 8) twiddles of the interpolating passes
  float4* wn_tw_col = nullptr;
  unsigned* wn_tiles = nullptr;             // (batch, ny) finished shares of a row tile, zero between passes
  float2* ttab = nullptr;                   // transmission table (draws, n_slices, ny, nx)
  size_t ttab_cap = 0;
  // buffers that a captured call reads: kept when larger ones take their places, until the plan goes
  bool ttab_captured = false, refs_captured = false;
  std::vector<void*> kept;
  wap::Detector det;                        // diffraction-pattern window (wap_plan_set_detector)
  unsigned long long* counter = nullptr;    // probe builder: aperture pixel count (allocated on first use)
  // a grid with an axis that is not a power of two: mixed-radix or Bluestein transforms
  bool generic = false;
  wap::GenAxis gen_x, gen_y;                // along x (rows) and y (columns)
  // one-launch chain of a single probe (wap_chain.cu): its twiddle table,
  // grid-barrier counter and status word (allocated on first use)
  float4* chain_tw = nullptr;
  int chain_e = 0;
  unsigned* chain_count = nullptr;
  int* chain_status = nullptr;
  int chain_ran = 0;                 // the last forward on this plan ran the chain kernel
  // cluster kernel (wap_cluster.cu): its (n, E) twiddle table, and whether the
  // device co-schedules a cluster of it (-1 not asked yet)
  float4* cl_tw = nullptr;
  int cl_e = 0;
  int cl_fits = -1;
};

namespace wap {

struct Physics {
  double e0, lambda, ri_a, ri_inv_den, kphase, k0, e_plus_e0;
};

Physics physics(double energy, double dz);
std::vector<float4> twiddle_table(int n, int e);

int fail(int code, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
void clear_error();
const char* last_error();

int check_common(const wap_plan* p, const float* V, int n_slices, int n_draws, const float* psi0, int n_probes,
                 float* exit);
// whether a stream is being captured: 1, 0, or -1 where the runtime will not say
int stream_capture(cudaStream_t st);
// gives up a buffer that a plan has outgrown: freed, or kept with the plan where a
// captured call holds its address
void drop_outgrown(wap_plan* p, void* d, bool captured);
// whether a kernel has to be allowed this much dynamic shared memory: 48 KB is the
// limit of dynamic and static together, and no kernel has 4 KB of static
inline bool beyond_default_smem(size_t dynamic) { return dynamic > 44 * 1024; }
int rows_per_cta(int nx, int e, int ny, int nb);
bool size_supported(int n);

struct RowArgs;
struct ColArgs;
struct WpmColArgs;
struct WpmRowArgs;
cudaError_t launch_row(int n, int e, const RowArgs& a, int nb, int k, cudaStream_t st);
cudaError_t launch_col(int n, int e, const ColArgs& a, int nb, int k, cudaStream_t st);
cudaError_t launch_wpm_col(int n, int e, const WpmColArgs& a, int nb, int k, cudaStream_t st);
cudaError_t launch_wpm_row(int n, int e, const WpmRowArgs& a, int nb, int k, cudaStream_t st);
// resident CTAs per SM of the WPM column (k = columns per CTA) and row (k = rows per CTA) kernels
int wpm_col_occupancy(int n, int e, int k, int K);
int wpm_row_occupancy(int n, int e, int k, int K);
cudaError_t row_chunks(const wap_plan* p, RowArgs r, int n_probes, cudaStream_t st);
cudaError_t col_chunks(const wap_plan* p, ColArgs c, int n_probes, cudaStream_t st);

// scheduler / chain overrides (wap_scan_debug_override), -1: default
int knob_value(int which);
// one-launch chain of a single probe (wap_chain.cu); returns -1 when the
// plan or the call does not qualify (the caller then launches per pass)
int chain_forward(wap_plan* p, const RowArgs& r, const ColArgs& c, int n_probes, int n_slices, float2* stack,
                  cudaStream_t st);
int cluster_forward(wap_plan* p, const RowArgs& r, const ColArgs& c, int n_probes, int n_slices, float2* stack,
                    cudaStream_t st);

// reference values and interpolation records of every slice (wap_wpm.cu)
struct WpmNodeScalars {
  bool sharing = false;   // slices without nodes may be shared out to more blocks
  bool nodes = false;   // records may hold interpolation nodes (else every slice forms its K reference fields)
  // the slope dz / (2 sqrt(qbar)) taken out per pixel, and qbar - k0^2, 1 / qbar, 1 / sqrt(qbar)
  float kappa = 0.f, dq = 0.f, inv_qbar = 0.f, inv_root_qbar = 0.f;
  float2 kk = {0.f, 0.f};   // kappa k0^2, hi and lo parts
};
int wpm_node_twiddles(wap_plan* p);

// grids that are not powers of two (wap_generic.cu)
bool generic_size_supported(int n);
int generic_axis_create(GenAxis* ax, int n);
void generic_axis_free(GenAxis* ax);
int generic_fresnel_forward(wap_plan* p, const RowArgs& r, const ColArgs& c, int n_slices, int n_probes,
                            float2* stack, cudaStream_t st);
cudaError_t gen_trans_table(const float* V, float2* ttab, long long n, const RowArgs& r, cudaStream_t st);
int generic_wpm_forward(const wap_plan* p, const WpmColArgs& c, const WpmRowArgs& w, const WpmNodeScalars& nodes,
                        double power, const float2* psi0, long long psi0_stride, const int32_t* positions,
                        int n_slices, int n_probes, float* dp, float2* stack, cudaStream_t st);
struct WpmNodeColArgs;
struct WpmNodeRowArgs;
WpmNodeColArgs wpm_node_col_args(const wap_plan* p, const WpmColArgs& c, const WpmNodeScalars& nodes);
WpmNodeRowArgs wpm_node_row_args(const wap_plan* p, const WpmRowArgs& w, const WpmNodeScalars& nodes, double power);
ColArgs base_col_args(const wap_plan* p, const float* H, const float* H_lo);
RowArgs base_row_args(const wap_plan* p, const Physics& ph, const float* V, int n_slices, const int32_t* draw);
int build_trans_table(wap_plan* p, const float* V, int n_slices, int n_draws, const RowArgs& r, cudaStream_t st);

// kernel-level tracing (wap_prof.cu)
struct ProfToken {
  bool active;
  int kind;
  cudaEvent_t a, b;
};
ProfToken prof_begin(int kind, cudaStream_t st);
void count_launch();  // every kernel launch of the library bumps wap_launch_count()
void prof_end(const ProfToken& t, cudaStream_t st, double bytes);

}  // namespace wap
