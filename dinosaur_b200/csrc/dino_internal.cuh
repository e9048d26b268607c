// Internal declarations shared by the dino_b200 CUDA sources.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>

#include <cstdio>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include "../../include/dino_b200.h"

namespace dino {

// ---------------------------------------------------------------------------
// Errors
// ---------------------------------------------------------------------------

void set_error(const std::string& msg);

struct Status {
  int code = DINO_OK;
};

#define DINO_CHECK_CUDA(expr)                                             \
  do {                                                                    \
    cudaError_t err_ = (expr);                                            \
    if (err_ != cudaSuccess) {                                            \
      ::dino::set_error(std::string(#expr) + ": " +                       \
                        cudaGetErrorString(err_));                        \
      return DINO_ERR_CUDA;                                               \
    }                                                                     \
  } while (0)

#define DINO_REQUIRE(cond, code, msg)        \
  do {                                       \
    if (!(cond)) {                           \
      ::dino::set_error(msg);                \
      return (code);                         \
    }                                        \
  } while (0)

#define DINO_TRY(expr)          \
  do {                          \
    int rc_ = (expr);           \
    if (rc_ != DINO_OK) return rc_; \
  } while (0)

// Checks the launch status of the last kernel (does not synchronize).
int check_launch(const char* what);

// Launches a kernel that may start while the one before it on the stream is
// finishing (programmatic dependent launch): its CTAs are brought up, and do
// what needs no earlier result, during the predecessor's last wave, which a
// plain launch would wait out.  Three rules hold for every kernel launched so:
//  - It calls pdl_wait() on every path before it touches memory that an earlier
//    kernel writes or reads, so it still sees the whole of its predecessor (and,
//    by the predecessor's own wait, of everything before it).
//  - If it takes something exclusive on its SM before pdl_wait() (TMEM), it calls
//    pdl_trigger() only once it holds it: no dependent CTA may exist while a
//    predecessor's CTA still has to get its share.
//  - It does not read a predecessor's results with __ldg or through const
//    __restrict__, which promise data that stays as it is for the whole of the
//    kernel and so may be read ahead of the wait; only a plan's tables are read so.
// Grids below kPdlMinCtas (less than two CTAs an SM of this chip) launch plainly:
// in a captured graph a programmatic edge between two short kernels costs more
// than the tail it hides (T21 / 12 steps 517 us plainly, 551 with every launch
// overlapped and 498 from 250 CTAs on; T85 shallow water 496, 620 and 497; T42 /
// 24 x 16 745, 725 and 725; TL159 pair of 75 fields 96.6, 89.0 and 88.9; moist
// TL255 / 32 x 4 11320, 11220 and 11180).
constexpr int64_t kPdlMinCtas = 250;
template <class... P, class... A>
int launch_pdl(const char* what, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
               cudaStream_t st, const A&... args) {
  static_assert(sizeof...(P) == sizeof...(A), "kernel arguments");
  std::tuple<std::remove_cv_t<P>...> values(args...);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = (int64_t)grid.x * grid.y * grid.z >= kPdlMinCtas ? 1 : 0;
  const cudaError_t err = std::apply(
      [&](auto&... v) {
        void* ptrs[] = {static_cast<void*>(&v)...};
        return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), ptrs);
      },
      values);
  if (err == cudaSuccess) return DINO_OK;
  cudaGetLastError();
  set_error(std::string("kernel launch failed (") + what + "): " + cudaGetErrorString(err));
  return DINO_ERR_CUDA;
}

// The kernel side of launch_pdl: lets the next kernel's CTAs come up (its own
// pdl_wait holds them until this grid has finished), and waits for the
// previous grid's end and memory.  Both are no-ops after a plain launch.
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A new device array with the values of src.  A copy from pageable memory may
// return before its last part has arrived, and a caller's non-blocking stream
// does not wait for the default one, so the copy is waited for.
template <typename T>
int upload(T** dst, const std::vector<T>& src) {
  DINO_CHECK_CUDA(cudaMalloc((void**)dst, sizeof(T) * (src.empty() ? 1 : src.size())));
  if (src.empty()) return DINO_OK;
  DINO_CHECK_CUDA(cudaMemcpy(*dst, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice));
  DINO_CHECK_CUDA(cudaStreamSynchronize(0));
  return DINO_OK;
}

// An NVTX range over the enclosing scope, so that profilers group the
// kernels a phase launches under the reference's names for its phases
// (inv_legendre, inv_fourier, fwd_fourier, fwd_legendre: the named calls of
// spherical_harmonic.py:265-279).  Costs nothing without an attached tool.
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange&) = delete;
  NvtxRange& operator=(const NvtxRange&) = delete;
};

// Runs a set-up step (returning a status) once per device and process, with
// that device current.  Kernel attributes such as the dynamic shared-memory
// limit belong to the device's context, so every device that launches the
// kernel needs its own call.  Safe to call from several host threads.
class PerDeviceOnce {
 public:
  template <class F>
  int run(F&& fn) {
    int dev = 0;
    DINO_CHECK_CUDA(cudaGetDevice(&dev));
    DINO_REQUIRE(dev >= 0 && dev < 64, DINO_ERR_ARG, "device index out of range");
    const uint64_t bit = 1ull << dev;
    std::lock_guard<std::mutex> lock(mu_);
    if (done_ & bit) return DINO_OK;
    DINO_TRY(fn());
    done_ |= bit;
    return DINO_OK;
  }

 private:
  std::mutex mu_;
  uint64_t done_ = 0;
};

// ---------------------------------------------------------------------------
// Field segments: a batch of fields gathered from up to kMaxSegs contiguous
// runs of [M][L] (or [I][J]) planes.
// ---------------------------------------------------------------------------

constexpr int kMaxSegs = 4;

struct Segs {
  const float* ptr[kMaxSegs];
  int start[kMaxSegs + 1];
  int n;
};

inline Segs one_seg(const float* p, int count) {
  Segs s{};
  s.ptr[0] = p;
  s.start[0] = 0;
  s.start[1] = count;
  s.n = 1;
  return s;
}

__device__ __forceinline__ const float* seg_field(const Segs& s, int b,
                                                  size_t stride) {
  int i = 0;
  while (i + 1 < s.n && b >= s.start[i + 1]) ++i;
  return s.ptr[i] + (size_t)(b - s.start[i]) * stride;
}

Segs seg_offset(const Segs& s, int first, int count, size_t stride);

// ---------------------------------------------------------------------------
// Transform plan
// ---------------------------------------------------------------------------

struct TcTables;  // tensor-core operand tables (legendre_tc.cu)

}  // namespace dino

struct dino_plan {
  // Shapes.
  int lw = 0, L = 0, I = 0, J = 0, M = 0, Jh = 0, N = 0;
  int spacing = 0, precision = 0, max_fields = 0, device = 0;
  int sms = 0;  // multiprocessors of the device
  double radius = 1.0;
  bool fft = false;  // I / 2 has a real FFT (else longitude sums are direct)
  // FP64 nodes and weights (device and host copies).
  double* d_x64 = nullptr;
  double* d_w64 = nullptr;
  std::vector<double> h_x64, h_w64;
  // FP32 tables.
  float* d_wq = nullptr;       // J: Gauss weight * 2pi / I
  float* d_ptab = nullptr;     // folded Legendre table, [m][l-m][Jh]
  int64_t* d_ptab_off = nullptr;  // lw + 1 offsets into d_ptab
  std::vector<int64_t> h_ptab_off;
  float* d_fbasis = nullptr;   // [I][M] real Fourier basis (generic DFT path)
  float2* d_tw_n = nullptr;    // N twiddles exp(+2 pi i k / N)
  float2* d_tw_i = nullptr;    // N twiddles exp(+2 pi i k / I)
  float* d_deriv = nullptr;    // 4 tables [lw][L]: (l+1)a, -l b, (l-1)a, -(l+2)b
  float* d_lap = nullptr;      // L: -l(l+1)/r^2
  float* d_invlap = nullptr;   // L: inverse, 0 at l = 0
  // Workspace: intermediate Fourier coefficients [max_fields][M][J].
  float* d_work = nullptr;
  dino::TcTables* tc = nullptr;
  // Second stream for alternating L2-sized chunks, with fork/join events.
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

namespace dino {

// ---------------------------------------------------------------------------
// Modal operators at one (row, l) of a [M][L] plane (real layout: rows
// m = 0, +1, -1, ...; deriv holds the recurrence tables of the plan).
// ---------------------------------------------------------------------------

// d/dlon: the cos/sin pair of each m swaps with a factor +-m.
__device__ __forceinline__ float d_dlon_at(const float* x, int row, int l,
                                           int L) {
  if (row == 0) return 0.f;
  int m = (row + 1) >> 1;
  return (row & 1) ? m * x[(size_t)(row + 1) * L + l]
                   : -m * x[(size_t)(row - 1) * L + l];
}

// cos_lat_d_dlat (tab = 0) or sec_lat_d_dlat_cos2 (tab = 2) at (row, l) of a
// plane x scaled elementwise by s[l] (s = nullptr: no scaling).
__device__ __forceinline__ float dlat_at(const float* x, const float* s,
                                         int row, int l, int L, int lw,
                                         const float* deriv, int tab) {
  int m = (row + 1) >> 1;
  const float* ta = deriv + (size_t)tab * lw * L + (size_t)m * L;
  const float* tb = ta + (size_t)lw * L;
  const float* xr = x + (size_t)row * L;
  float v = 0.f;
  if (l + 1 < L) v += ta[l + 1] * (s ? s[l + 1] * xr[l + 1] : xr[l + 1]);
  if (l >= 1) v += tb[l - 1] * (s ? s[l - 1] * xr[l - 1] : xr[l - 1]);
  return v;
}

// sht.cu
int sht_inverse_segs(dino_plan* p, const Segs& in, float* out_nodal, int nfields,
                     float* work, int work_fields, cudaStream_t st);
int sht_forward_to(dino_plan* p, const float* nodal, float* out_modal,
                   int nfields, float* work, int work_fields, cudaStream_t st);
int sht_inverse_adjoint_to(dino_plan* p, const float* nodal_ct, float* modal_ct,
                           int nfields, float* work, int work_fields, cudaStream_t st);
int sht_forward_adjoint_to(dino_plan* p, const float* modal_ct, float* nodal_ct,
                           int nfields, float* work, int work_fields, cudaStream_t st);
// Fields per chunk of a chunked transform of nf fields (sht.cu).
int l2_chunk(dino_plan* p, int nf, int work_fields);
int legendre_inverse(dino_plan* p, const Segs& in, float* out_fourier,
                     int nfields, cudaStream_t st);
int legendre_forward(dino_plan* p, const float* fourier, float* out_modal,
                     int nfields, cudaStream_t st);
int fourier_inverse(dino_plan* p, const float* fourier, float* nodal,
                    int nfields, bool weighted_adjoint, cudaStream_t st);
int fourier_forward(dino_plan* p, const float* nodal, float* fourier,
                    int nfields, bool weighted, cudaStream_t st);
int modal_op(dino_plan* p, int op, const float* in, float* out, int nfields,
             int arg, cudaStream_t st);
// Whether the real FFT covers a half length I / 2 = n.
bool fft_supported(int n);
// Sets kernel attributes ahead of stream capture.
int sht_prepare(dino_plan* p);
// FP32 SIMT inverse Legendre contraction for any plan (no precision dispatch).
std::string tc_describe(dino_plan* p);  // legendre_tc.cu
int legendre_inverse_fp32(dino_plan* p, const Segs& in, float* out, int nf,
                          cudaStream_t st);
// FP32 SIMT forward Legendre contraction for any plan.
int legendre_forward_fp32(dino_plan* p, const float* fourier, float* out, int nf,
                          cudaStream_t st);
// Whether a tensor-core plan's autotuner found the FP32 SIMT contraction of
// this direction faster at its chunk size (legendre_tc.cu).
bool tc_use_simt(const dino_plan* p, bool forward);

// legendre_tc.cu
int tc_tables_build(dino_plan* p);
void tc_tables_free(dino_plan* p);
int tc_legendre_inverse(dino_plan* p, const Segs& in, float* out_fourier,
                        int nfields, cudaStream_t st);
int tc_legendre_forward(dino_plan* p, const float* fourier, float* out_modal,
                        int nfields, cudaStream_t st);

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

}  // namespace dino
