// Shallow-water equations on the sphere: explicit tendencies, implicit terms
// and the closed-form implicit inverse (ShallowWaterEquations,
// dinosaur/shallow_water.py:121-230).
//
// Packed state, kind-major: [vorticity: members*K][divergence][potential]
// planes of [M][L].  One explicit evaluation is
//   modal pre-pass (u cos, v cos, clipped vorticity and potential)
//   -> inverse SHT -> nodal products (u (zeta + f), u phi, kinetic energy)
//   -> forward SHT -> modal post-pass (div/curl, Laplacian, the layer
//   pressure coupling through the density ratios, clip of the top l).
// A filtered SIL3 step is three of them, the post-pass of each fused with the
// stage that follows (the implicit part is elementwise in (layer, m, l)): 21
// kernels, replayed from one CUDA graph, in place of about 150 launches of the
// generic tableau loop over tensors, which the host could not issue as fast as
// the GPU ran them.

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <mutex>
#include <vector>

#include "dino_internal.cuh"

struct dino_swe {
  dino_plan* plan = nullptr;
  int K = 0, mem = 0, M = 0, L = 0, I = 0, J = 0;
  size_t ML = 0, IJ = 0;
  float* d_dens = nullptr;   // K x K density ratios (shallow_water.py:71-86)
  float* d_phiref = nullptr; // K reference potentials
  float* d_orog = nullptr;   // [M][L] modal orography (zeros when absent)
  float* d_lat = nullptr;    // [2][J]: sec^2(lat), 2 Omega sin(lat)
  float* d_aux = nullptr;    // [u][v][zeta clipped][phi clipped]: 4 mK planes
  float* d_nodal = nullptr;  // their nodal values
  float* d_fwd_in = nullptr; // [b_u][b_v][g_u][g_v][e]: 5 mK nodal planes
  float* d_fwd_out = nullptr;
  float* d_work = nullptr;
  int work_fields = 0;
  // SIL3 step (allocated by the first one): the state it advances, the two
  // stage states, f0 and f1, and the captured steps.
  float* d_y = nullptr;
  float* d_Y[2] = {nullptr, nullptr};
  float* d_f[2] = {nullptr, nullptr};
  // The captured step of one time step and filter (empty: none), with the
  // filter on the device.  Calls take turns between a few of them (a forward and
  // a backward sweep, a halved time step); the least recently used goes.
  struct Step {
    double dt = 0;
    std::vector<double> host_filter;
    float* d_filter = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t used = 0;
  };
  static constexpr size_t kMaxSteps = 8;
  std::vector<Step> steps;
  uint64_t calls = 0;
  std::mutex mu;  // held while a step is found and queued
};

namespace dino {
namespace {

struct SwePrepArgs {
  const float* state;
  float* aux;
  int K, mem, M, L, lw;
  const float* deriv;
  const float* invlap;
  float inv_radius;
};

// get_cos_lat_vector(vorticity, divergence, grid) with its default clip
// (spherical_harmonic.py:1164-1178) and clip_wavenumbers of vorticity and
// potential before their inverse transforms (shallow_water.py:60-62).
__global__ void swe_prep_kernel(SwePrepArgs a) {
  pdl_trigger();
  pdl_wait();
  const size_t ML = (size_t)a.M * a.L;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ML) return;
  const int l = idx % a.L, row = idx / a.L;
  const size_t mK = (size_t)a.mem * a.K;
  const size_t plane = (size_t)blockIdx.z * a.K + blockIdx.y;  // member, level
  const float* vort = a.state + plane * ML;
  const float* div = a.state + (mK + plane) * ML;
  const float* phi = a.state + (2 * mK + plane) * ML;
  const bool keep = l < a.L - 1;
  float u = 0.f, v = 0.f;
  if (keep) {
    const float dchi = d_dlon_at(div, row, l, a.L) * a.invlap[l];
    const float dpsi = d_dlon_at(vort, row, l, a.L) * a.invlap[l];
    const float cchi = dlat_at(div, a.invlap, row, l, a.L, a.lw, a.deriv, 0);
    const float cpsi = dlat_at(vort, a.invlap, row, l, a.L, a.lw, a.deriv, 0);
    u = (dchi - cpsi) * a.inv_radius;
    v = (cchi + dpsi) * a.inv_radius;
  }
  a.aux[plane * ML + idx] = u;
  a.aux[(mK + plane) * ML + idx] = v;
  a.aux[(2 * mK + plane) * ML + idx] = keep ? vort[idx] : 0.f;
  a.aux[(3 * mK + plane) * ML + idx] = keep ? phi[idx] : 0.f;
}

struct SweNodalArgs {
  const float* nod;  // [u][v][zeta][phi]
  float* fwd;        // [b_u][b_v][g_u][g_v][e]
  int J;
  size_t IJ, mK;
  const float* lat;
};

// shallow_water.py:170-177: b = u (zeta + f) sec^2, g = u phi sec^2,
// e = |u|^2 sec^2 / 2 on the nodal grid.
__global__ void swe_nodal_kernel(SweNodalArgs a) {
  pdl_trigger();
  pdl_wait();
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= a.IJ) return;
  const size_t plane = blockIdx.y;
  const int j = idx % a.J;
  const float sec2 = a.lat[j];
  const float f = a.lat[a.J + j];
  const size_t s = a.mK * a.IJ, o = plane * a.IJ + idx;
  const float u = a.nod[o], v = a.nod[s + o];
  const float tv = a.nod[2 * s + o] + f;
  const float phi = a.nod[3 * s + o];
  a.fwd[o] = u * tv * sec2;
  a.fwd[s + o] = v * tv * sec2;
  a.fwd[2 * s + o] = u * phi * sec2;
  a.fwd[3 * s + o] = v * phi * sec2;
  a.fwd[4 * s + o] = (u * u + v * v) * sec2 * 0.5f;
}

struct SwePostArgs {
  const float* fm;     // modal [b_u][b_v][g_u][g_v][e]
  const float* state;  // for the potential
  float* tend;
  const float* dens;   // K x K
  const float* orog;
  int K, mem, M, L, lw;
  const float* deriv;
  const float* lap;
  float inv_radius;
};

// The tendencies of one (member, layer, row, l) (shallow_water.py:186-205).
// p = D phi + orography (the layers' pressure coupling); vorticity
// -div_cos_lat(b); divergence -lap(p + e) + curl_cos_lat(b); potential
// -div_cos_lat(g); every tendency clipped.
__device__ __forceinline__ void swe_tendency(const SwePostArgs& a, int mb, int k, size_t idx,
                                             float& fz, float& fd, float& fp) {
  const size_t ML = (size_t)a.M * a.L;
  const int l = idx % a.L, row = idx / a.L, K = a.K;
  fz = fd = fp = 0.f;
  if (l == a.L - 1) return;
  const size_t mK = (size_t)a.mem * K;
  const size_t plane = (size_t)mb * K + k;
  const float* bu = a.fm + plane * ML;
  const float* bv = a.fm + (mK + plane) * ML;
  const float* gu = a.fm + (2 * mK + plane) * ML;
  const float* gv = a.fm + (3 * mK + plane) * ML;
  const float* e = a.fm + (4 * mK + plane) * ML;
  const float ir = a.inv_radius;
  float p = a.orog[idx];
  for (int b = 0; b < K; ++b)
    p = fmaf(a.dens[k * K + b], a.state[(2 * mK + (size_t)mb * K + b) * ML + idx], p);
  const float div_b = (d_dlon_at(bu, row, l, a.L) +
                       dlat_at(bv, nullptr, row, l, a.L, a.lw, a.deriv, 2)) * ir;
  const float curl_b = (d_dlon_at(bv, row, l, a.L) -
                        dlat_at(bu, nullptr, row, l, a.L, a.lw, a.deriv, 2)) * ir;
  const float div_g = (d_dlon_at(gu, row, l, a.L) +
                       dlat_at(gv, nullptr, row, l, a.L, a.lw, a.deriv, 2)) * ir;
  fz = -div_b;
  fd = -a.lap[l] * (p + e[idx]) + curl_b;
  fp = -div_g;
}

__global__ void swe_post_kernel(SwePostArgs a) {
  pdl_trigger();
  pdl_wait();
  const size_t ML = (size_t)a.M * a.L;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ML) return;
  const int k = blockIdx.y, mb = blockIdx.z;
  const size_t mK = (size_t)a.mem * a.K;
  const size_t plane = (size_t)mb * a.K + k;
  float fz, fd, fp;
  swe_tendency(a, mb, k, idx, fz, fd, fp);
  a.tend[plane * ML + idx] = fz;
  a.tend[(mK + plane) * ML + idx] = fd;
  a.tend[(2 * mK + plane) * ML + idx] = fp;
}

// Stage kStage (1, 2, 3) of a filtered SIL3 step (time_integration.py:329-405)
// from the transform outputs of its explicit evaluation at a.state (y0, Y1 or
// Y2): the tendency f, the combination with y0, the earlier f_j and the
// implicit terms (elementwise in (layer, m, l), so they are formed here from
// the states themselves), the implicit inverse, and in the last stage the
// final implicit term and the filter.  a.tend (stages 1, 2): where f is kept.
struct SweStageArgs {
  const float* y0;
  const float* f0;
  const float* f1;
  float* out;
  const float* phiref;
  const float* filter;  // per l, or null (last stage)
  float c0, c1, cf;     // coefficients of f0, f1 and f
  float cg, eta;        // of the implicit terms, and of the implicit inverse
};

template <int kStage>
__global__ void swe_stage_kernel(SwePostArgs a, SweStageArgs s) {
  pdl_trigger();
  pdl_wait();
  const size_t ML = (size_t)a.M * a.L;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= ML) return;
  const int l = idx % a.L, k = blockIdx.y, mb = blockIdx.z;
  const size_t mK = (size_t)a.mem * a.K;
  const size_t plane = (size_t)mb * a.K + k;
  const size_t oz = plane * ML + idx, od = (mK + plane) * ML + idx,
               op = (2 * mK + plane) * ML + idx;
  float fz, fd, fp;
  swe_tendency(a, mb, k, idx, fz, fd, fp);
  if (kStage < 3) {
    a.tend[oz] = fz;
    a.tend[od] = fd;
    a.tend[op] = fp;
  }
  const float lam = a.lap[l], ref = s.phiref[k];
  const float y0d = s.y0[od], y0p = s.y0[op];
  float z = s.y0[oz], d = y0d, p = y0p;
  auto add = [&](float c, float vz, float vd, float vp) {
    z = fmaf(c, vz, z);
    d = fmaf(c, vd, d);
    p = fmaf(c, vp, p);
  };
  if (kStage > 1) add(s.c0, s.f0[oz], s.f0[od], s.f0[op]);
  if (kStage > 2) add(s.c1, s.f1[oz], s.f1[od], s.f1[op]);
  add(s.cf, fz, fd, fp);
  // g0 (and g2 at Y2 = a.state).
  add(s.cg, 0.f, -lam * y0p, -ref * y0d);
  if (kStage == 3) add(s.cg, 0.f, -lam * a.state[op], -ref * a.state[od]);
  const float eta = s.eta;
  const float inv = 1.f / (1.f - eta * eta * ref * lam);
  const float sd = inv * (d - eta * lam * p);
  const float sp = inv * (p - eta * ref * d);
  if (kStage < 3) {
    s.out[oz] = z;
    s.out[od] = sd;
    s.out[op] = sp;
  } else {
    const float w = s.filter ? s.filter[l] : 1.f;
    s.out[oz] = z * w;
    s.out[od] = fmaf(eta, -lam * sp, d) * w;
    s.out[op] = fmaf(eta, -ref * sd, p) * w;
  }
}

struct SweImplicitArgs {
  const float* in;
  float* out;
  const float* phiref;
  const float* lap;
  float eta;
  int mode;  // 0: implicit terms, 1: implicit inverse
  int K, mem, L;
  size_t ML;
};

// shallow_water.py:207-230, elementwise per (layer, m, l).
__global__ void swe_implicit_kernel(SweImplicitArgs a) {
  pdl_trigger();
  pdl_wait();
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= a.ML) return;
  const int l = idx % a.L;
  const int k = blockIdx.y, mb = blockIdx.z;
  const size_t mK = (size_t)a.mem * a.K;
  const size_t plane = (size_t)mb * a.K + k;
  const size_t oz = plane * a.ML + idx, od = (mK + plane) * a.ML + idx,
               op = (2 * mK + plane) * a.ML + idx;
  const float z = a.in[oz], d = a.in[od], p = a.in[op];
  const float lam = a.lap[l], ref = a.phiref[k];
  if (a.mode == 0) {
    a.out[oz] = 0.f;
    a.out[od] = -lam * p;
    a.out[op] = -ref * d;
  } else {
    const float s = 1.f / (1.f - a.eta * a.eta * ref * lam);
    a.out[oz] = z;
    a.out[od] = s * (d - a.eta * lam * p);
    a.out[op] = s * (-a.eta * ref * d + p);
  }
}

void step_free(dino_swe::Step* g) {
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  cudaFree(g->d_filter);
}

void swe_free(dino_swe* s) {
  if (!s) return;
  cudaFree(s->d_dens);
  cudaFree(s->d_phiref);
  cudaFree(s->d_orog);
  cudaFree(s->d_lat);
  cudaFree(s->d_aux);
  cudaFree(s->d_nodal);
  cudaFree(s->d_fwd_in);
  cudaFree(s->d_fwd_out);
  cudaFree(s->d_work);
  for (auto& g : s->steps) step_free(&g);
  cudaFree(s->d_y);
  for (float* b : s->d_Y) cudaFree(b);
  for (float* b : s->d_f) cudaFree(b);
  delete s;
}

int swe_build(dino_swe* s, const dino_swe_desc* d) {
  dino_plan* p = s->plan;
  const int K = s->K;
  std::vector<float> dens(K * K), ref(K), lat(2 * p->J);
  // D[i][j] = min(rho_j / rho_i, 1) with a zero diagonal: the pressure on
  // layer i from the layers j (shallow_water.py:71-86).
  for (int i = 0; i < K; ++i) {
    for (int j = 0; j < K; ++j) {
      const double r = d->densities ? d->densities[j] / d->densities[i] : 1.0;
      dens[i * K + j] = (i == j) ? 0.f : (float)(r < 1.0 ? r : 1.0);
    }
    ref[i] = (float)d->reference_potential[i];
  }
  for (int j = 0; j < p->J; ++j) {
    const double x = p->h_x64[j];
    lat[j] = (float)(1.0 / (1.0 - x * x));
    lat[p->J + j] = (float)(2.0 * d->angular_velocity * x);
  }
  DINO_TRY(upload(&s->d_dens, dens));
  DINO_TRY(upload(&s->d_phiref, ref));
  DINO_TRY(upload(&s->d_lat, lat));
  std::vector<float> orog(s->ML, 0.f);
  if (d->orography_modal)
    for (size_t i = 0; i < s->ML; ++i) orog[i] = d->orography_modal[i];
  DINO_TRY(upload(&s->d_orog, orog));
  const size_t mK = (size_t)s->mem * K;
  DINO_CHECK_CUDA(cudaMalloc(&s->d_aux, sizeof(float) * 4 * mK * s->ML));
  DINO_CHECK_CUDA(cudaMalloc(&s->d_nodal, sizeof(float) * 4 * mK * s->IJ));
  DINO_CHECK_CUDA(cudaMalloc(&s->d_fwd_in, sizeof(float) * 5 * mK * s->IJ));
  DINO_CHECK_CUDA(cudaMalloc(&s->d_fwd_out, sizeof(float) * 5 * mK * s->ML));
  s->work_fields = (int)(5 * mK);
  DINO_CHECK_CUDA(cudaMalloc(&s->d_work, sizeof(float) * 5 * mK * p->M * p->J));
  return DINO_OK;
}

// The explicit terms of `state` up to the forward transform (s->d_fwd_out).
int swe_products(dino_swe* s, const float* state, cudaStream_t st) {
  dino_plan* p = s->plan;
  const int K = s->K, mem = s->mem;
  const int mK = mem * K;
  {
    SwePrepArgs a{state, s->d_aux, K, mem, s->M, s->L, p->lw, p->d_deriv, p->d_invlap,
                  (float)(1.0 / p->radius)};
    dim3 grid(ceil_div((int)s->ML, 256), K, mem);
    DINO_TRY(launch_pdl("swe_prep", swe_prep_kernel, grid, 256, 0, st, a));
  }
  DINO_TRY(sht_inverse_segs(p, one_seg(s->d_aux, 4 * mK), s->d_nodal, 4 * mK, s->d_work,
                            s->work_fields, st));
  {
    SweNodalArgs a{s->d_nodal, s->d_fwd_in, s->J, s->IJ, (size_t)mK, s->d_lat};
    dim3 grid(ceil_div((int)s->IJ, 256), mK);
    DINO_TRY(launch_pdl("swe_nodal", swe_nodal_kernel, grid, 256, 0, st, a));
  }
  return sht_forward_to(p, s->d_fwd_in, s->d_fwd_out, 5 * mK, s->d_work, s->work_fields, st);
}

SwePostArgs post_args(dino_swe* s, const float* state, float* tend) {
  return {s->d_fwd_out, state, tend, s->d_dens, s->d_orog, s->K, s->mem, s->M, s->L,
          s->plan->lw, s->plan->d_deriv, s->plan->d_lap, (float)(1.0 / s->plan->radius)};
}

int swe_explicit_impl(dino_swe* s, const float* state, float* tend, cudaStream_t st) {
  DINO_TRY(swe_products(s, state, st));
  dim3 grid(ceil_div((int)s->ML, 256), s->K, s->mem);
  return launch_pdl("swe_post", swe_post_kernel, grid, 256, 0, st, post_args(s, state, tend));
}

// One filtered SIL3 step of s->d_y in place.
int swe_step_once(dino_swe* s, double dt, const float* filter, cudaStream_t st) {
  dim3 grid(ceil_div((int)s->ML, 256), s->K, s->mem);
  SweStageArgs a{};
  a.y0 = s->d_y;
  a.f0 = s->d_f[0];
  a.f1 = s->d_f[1];
  a.phiref = s->d_phiref;
  DINO_TRY(swe_products(s, s->d_y, st));
  a.out = s->d_Y[0];
  a.cf = (float)(dt / 3);
  a.cg = a.eta = (float)(dt / 6);
  DINO_TRY(launch_pdl("swe_stage", swe_stage_kernel<1>, grid, 256, 0, st,
                      post_args(s, s->d_y, s->d_f[0]), a));
  DINO_TRY(swe_products(s, s->d_Y[0], st));
  a.out = s->d_Y[1];
  a.c0 = (float)(dt / 6);
  a.cf = (float)(dt / 2);
  a.cg = a.eta = (float)(dt / 3);
  DINO_TRY(launch_pdl("swe_stage", swe_stage_kernel<2>, grid, 256, 0, st,
                      post_args(s, s->d_Y[0], s->d_f[1]), a));
  DINO_TRY(swe_products(s, s->d_Y[1], st));
  a.out = s->d_y;
  a.filter = filter;
  a.c0 = (float)(dt / 2);
  a.c1 = (float)(-dt / 2);
  a.cf = (float)dt;
  a.cg = (float)(3 * dt / 8);
  a.eta = (float)(dt / 4);
  return launch_pdl("swe_stage", swe_stage_kernel<3>, grid, 256, 0, st,
                    post_args(s, s->d_Y[1], nullptr), a);
}

// Uploads the filter and captures the step of g.
int swe_capture(dino_swe* s, dino_swe::Step* g) {
  if (!g->host_filter.empty())
    DINO_TRY(upload(&g->d_filter,
                    std::vector<float>(g->host_filter.begin(), g->host_filter.end())));
  DINO_TRY(sht_prepare(s->plan));
  // Captured on a private stream, so that the caller's stream (possibly the
  // legacy default one) never enters capture mode.
  cudaStream_t cap;
  DINO_CHECK_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
  cudaError_t ce = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  int rc = DINO_OK;
  if (ce == cudaSuccess) {
    rc = swe_step_once(s, g->dt, g->d_filter, cap);
    ce = cudaStreamEndCapture(cap, &g->graph);
  }
  cudaStreamDestroy(cap);
  if (rc != DINO_OK) return rc;
  DINO_CHECK_CUDA(ce);
  ce = cudaGraphInstantiate(&g->exec, g->graph, 0);
  if (ce != cudaSuccess) g->exec = nullptr;
  DINO_CHECK_CUDA(ce);
  return DINO_OK;
}

// The captured step of (dt, filter), captured now if it is not among the last.
int swe_find_step(dino_swe* s, double dt, const double* host_filter, cudaGraphExec_t* exec) {
  const size_t n = host_filter ? (size_t)s->L : 0;
  for (auto& g : s->steps)
    if (g.dt == dt && g.host_filter.size() == n &&
        (n == 0 || std::memcmp(g.host_filter.data(), host_filter, sizeof(double) * n) == 0)) {
      g.used = ++s->calls;
      *exec = g.exec;
      return DINO_OK;
    }
  dino_swe::Step g;
  g.dt = dt;
  if (n) g.host_filter.assign(host_filter, host_filter + n);
  s->steps.reserve(dino_swe::kMaxSteps);
  const int rc = swe_capture(s, &g);
  if (rc != DINO_OK) {
    step_free(&g);
    return rc;
  }
  g.used = ++s->calls;
  *exec = g.exec;
  if (s->steps.size() < dino_swe::kMaxSteps) {
    s->steps.push_back(std::move(g));
    return DINO_OK;
  }
  auto old = std::min_element(s->steps.begin(), s->steps.end(),
                              [](const auto& a, const auto& b) { return a.used < b.used; });
  // Its last launch may still be queued and read its filter.
  DINO_CHECK_CUDA(cudaDeviceSynchronize());
  step_free(&*old);
  *old = std::move(g);
  return DINO_OK;
}

int swe_step_impl(dino_swe* s, float* state, double dt, const double* host_filter, int n_steps,
                  cudaStream_t st) {
  std::lock_guard<std::mutex> lock(s->mu);
  const size_t bytes = sizeof(float) * 3 * (size_t)s->mem * s->K * s->ML;
  for (float** b : {&s->d_y, &s->d_Y[0], &s->d_Y[1], &s->d_f[0], &s->d_f[1]})
    if (!*b) DINO_CHECK_CUDA(cudaMalloc(b, bytes));
  cudaGraphExec_t exec = nullptr;
  DINO_TRY(swe_find_step(s, dt, host_filter, &exec));
  // The captured step works on the object's own buffer, so one capture serves
  // every caller's state; two copies a call.
  DINO_CHECK_CUDA(cudaMemcpyAsync(s->d_y, state, bytes, cudaMemcpyDeviceToDevice, st));
  for (int i = 0; i < n_steps; ++i) DINO_CHECK_CUDA(cudaGraphLaunch(exec, st));
  DINO_CHECK_CUDA(cudaMemcpyAsync(state, s->d_y, bytes, cudaMemcpyDeviceToDevice, st));
  return DINO_OK;
}

int swe_implicit_impl(dino_swe* s, const float* in, float* out, int mode, double eta,
                      cudaStream_t st) {
  SweImplicitArgs a{in, out, s->d_phiref, s->plan->d_lap, (float)eta, mode, s->K, s->mem,
                    s->L, s->ML};
  dim3 grid(ceil_div((int)s->ML, 256), s->K, s->mem);
  return launch_pdl("swe_implicit", swe_implicit_kernel, grid, 256, 0, st, a);
}

}  // namespace
}  // namespace dino

using namespace dino;

extern "C" {

int dino_swe_create(dino_plan* plan, const dino_swe_desc* d, dino_swe** out) {
  DINO_REQUIRE(plan && d && out, DINO_ERR_ARG, "dino_swe_create: null argument");
  DINO_REQUIRE(d->layers >= 1 && d->layers <= 256, DINO_ERR_UNSUPPORTED,
               "layers must be in [1, 256]");
  DINO_REQUIRE(d->members >= 1, DINO_ERR_ARG, "members must be >= 1");
  DINO_REQUIRE(d->reference_potential != nullptr, DINO_ERR_ARG,
               "dino_swe_create: missing reference potential");
  if (d->densities)
    for (int i = 0; i < d->layers; ++i)
      DINO_REQUIRE(d->densities[i] > 0, DINO_ERR_ARG, "densities must be positive");
  dino_swe* s = new dino_swe();
  s->plan = plan;
  s->K = d->layers;
  s->mem = d->members;
  s->M = plan->M;
  s->L = plan->L;
  s->I = plan->I;
  s->J = plan->J;
  s->ML = (size_t)s->M * s->L;
  s->IJ = (size_t)s->I * s->J;
  const int rc = swe_build(s, d);
  if (rc != DINO_OK) {
    swe_free(s);
    return rc;
  }
  *out = s;
  return DINO_OK;
}

int dino_swe_destroy(dino_swe* s) {
  swe_free(s);
  return DINO_OK;
}

int64_t dino_swe_state_size(const dino_swe* s) {
  return s ? (int64_t)3 * s->mem * s->K * (int64_t)s->ML : -1;
}

int dino_swe_explicit(dino_swe* s, const float* state, float* out, void* stream) {
  DINO_REQUIRE(s && state && out, DINO_ERR_ARG, "dino_swe_explicit: null argument");
  DINO_REQUIRE(state != out, DINO_ERR_ARG, "dino_swe_explicit: in and out must differ");
  return swe_explicit_impl(s, state, out, (cudaStream_t)stream);
}

int dino_swe_implicit(dino_swe* s, const float* state, float* out, void* stream) {
  DINO_REQUIRE(s && state && out, DINO_ERR_ARG, "dino_swe_implicit: null argument");
  return swe_implicit_impl(s, state, out, 0, 0.0, (cudaStream_t)stream);
}

int dino_swe_implicit_inverse(dino_swe* s, const float* state, float* out, double eta,
                              void* stream) {
  DINO_REQUIRE(s && state && out, DINO_ERR_ARG, "dino_swe_implicit_inverse: null argument");
  DINO_REQUIRE(std::isfinite(eta), DINO_ERR_ARG, "step_size must be finite");
  return swe_implicit_impl(s, state, out, 1, eta, (cudaStream_t)stream);
}

int dino_swe_step(dino_swe* s, float* state, double dt, const double* host_filter,
                  int32_t n_steps, void* stream) {
  DINO_REQUIRE(s && state, DINO_ERR_ARG, "dino_swe_step: null argument");
  DINO_REQUIRE(n_steps >= 0, DINO_ERR_ARG, "n_steps must be >= 0");
  if (n_steps == 0) return DINO_OK;
  DINO_REQUIRE(std::isfinite(dt), DINO_ERR_ARG, "step_size must be finite");
  try {
    return swe_step_impl(s, state, dt, host_filter, n_steps, (cudaStream_t)stream);
  } catch (const std::exception& e) {
    set_error(std::string("dino_swe_step: ") + e.what());
    return DINO_ERR_CUDA;
  }
}

}  // extern "C"
