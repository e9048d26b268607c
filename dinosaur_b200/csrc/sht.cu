// Spherical-harmonic transform pair on one B200: per-m Legendre contraction
// over Gaussian latitude (N/S folded, FP32 SIMT form here; tensor-core form in
// legendre_tc.cu) and a real FFT over longitude in shared memory.
//
// Semantics follow RealSphericalHarmonics.inverse_transform / transform
// (dinosaur/spherical_harmonic.py:262-280):
//   inverse:  px[b,m,j] = sum_l p[m,j,l] x[b,m,l];  out[b,i,j] = sum_m f[i,m] px[b,m,j]
//   forward:  fwx[b,m,j] = sum_i f[i,m] w[j] z[b,i,j];  out[b,m,l] = sum_j p[m,j,l] fwx[b,m,j]
// with f the unit-norm real Fourier basis (fourier.py:24-60) and p the
// normalised associated Legendre functions duplicated over +-m rows.
//
// Folding: Gauss nodes are mirror symmetric and p[m, J-1-j, l] =
// (-1)^(l-m) p[m, j, l], so each contraction splits into even and odd (l-m)
// halves over Jh = ceil(J/2) latitudes, halving the arithmetic.

#include <cmath>

#include <algorithm>

#include "dino_internal.cuh"

namespace dino {

// ---------------------------------------------------------------------------
// Legendre contraction, FP32 SIMT
// ---------------------------------------------------------------------------

// A CTA has TB (field, cos/sin) rows and as many threads: 128, or 64 for short
// batches (leg_rows).
constexpr int kLegTN = 32;   // latitudes (inverse) per CTA
constexpr int kLegKC = 16;   // contraction chunk

// Row r of the m-slice: m == 0 has one row per field (cos), m > 0 has two.
__device__ __forceinline__ void row_map(int m, int r, int& b, int& row) {
  if (m == 0) {
    b = r;
    row = 0;
  } else {
    b = r >> 1;
    row = 2 * m - 1 + (r & 1);
  }
}

// Each thread stages 4 rows x 4 contraction indices of a TB x 16 operand
// chunk: rows (tid / 4) + TB / 4 i, indices 4 (tid % 4) .. + 3.  Row pointers are
// resolved once per CTA; the next chunk is prefetched into registers while
// the current one is consumed from shared memory.

// out_fourier[b][row][j] for all j from modal rows (inverse contraction).  Two
// rows share an f32x2 FMA: the loop was bound by its issue slots and its
// shared-memory reads together, and a value's place in two registers is free.
// The bound of three CTAs of 128 an SM keeps the accumulators in registers (the
// 64-row form spills two other values; with four CTAs the accumulators spill:
// TL255, 64 fields 56 us).  TL159, 75 fields 26.0 -> 24.4 us, TL255,
// 64 fields 42.4 -> 40.1, T42, 900 fields 11.6 -> 10.5.
template <int TB>
__global__ void __launch_bounds__(TB, 3 * 128 / TB)
legendre_inverse_simt(Segs in, float* __restrict__ out, int B, int M, int L,
                      int J, int Jh, const float* __restrict__ ptab,
                      const int64_t* __restrict__ ptab_off) {
  pdl_trigger();
  pdl_wait();
  const int m = blockIdx.z;
  const int rows = (m == 0) ? B : 2 * B;
  const int r0 = blockIdx.y * TB;
  if (r0 >= rows) return;
  const int j0 = blockIdx.x * kLegTN;
  const int Lm = L - m;
  const float* P = ptab + ptab_off[m];

  __shared__ __align__(16) float Xs[kLegKC][TB + 4];
  __shared__ __align__(16) float Ps[kLegKC][kLegTN];

  const int tid = threadIdx.x;
  const int tx = tid & 7;   // 8 groups of 4 latitudes
  const int ty = tid >> 3;  // 16 groups of 8 rows
  const int lq = tid & 3;   // load quarter (4 contraction indices)
  const float* xrow[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + (tid >> 2) + TB / 4 * i;
    xrow[i] = nullptr;
    if (r < rows) {
      int b, row;
      row_map(m, r, b, row);
      xrow[i] = seg_field(in, b, (size_t)M * L) + (size_t)row * L + m;
    }
  }
  constexpr int kPv = 128 / TB;  // float4 of the 16 x 32 table chunk per thread
  const int pk = tid >> 3, pj = (tid & 7) * 4;
  float xv[4][4];
  float4 pv[kPv];
  auto fetch = [&](int kc) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = kc + lq * 4 + e;
        xv[i][e] = (xrow[i] && k < Lm) ? xrow[i][k] : 0.f;
      }
#pragma unroll
    for (int i = 0; i < kPv; ++i) {
      const int k = kc + pk + TB / 8 * i;
      const int j = j0 + pj;
      // Vector load only when the row start is 16-byte aligned (Jh % 4 == 0;
      // the per-m table offsets are multiples of Jh).
      if ((Jh & 3) == 0 && k < Lm && j + 3 < Jh) {
        pv[i] = *reinterpret_cast<const float4*>(P + (size_t)k * Jh + j);
      } else {
        float t[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          t[e] = (k < Lm && j + e < Jh) ? P[(size_t)k * Jh + j + e] : 0.f;
        pv[i] = make_float4(t[0], t[1], t[2], t[3]);
      }
    }
  };

  float2 aE[4][4], aO[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int t = 0; t < 4; ++t) aE[i][t] = aO[i][t] = make_float2(0.f, 0.f);

  fetch(0);
  for (int kc = 0; kc < Lm; kc += kLegKC) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) Xs[lq * 4 + e][(tid >> 2) + TB / 4 * i] = xv[i][e];
#pragma unroll
    for (int i = 0; i < kPv; ++i)
      *reinterpret_cast<float4*>(&Ps[pk + TB / 8 * i][pj]) = pv[i];
    __syncthreads();
    if (kc + kLegKC < Lm) fetch(kc + kLegKC);
#pragma unroll
    for (int kk = 0; kk < kLegKC; kk += 2) {
      auto step = [&](int k, float2 (&acc)[4][4]) {
        const float4 xa = *reinterpret_cast<const float4*>(&Xs[k][ty * 8]);
        const float4 xb = *reinterpret_cast<const float4*>(&Xs[k][ty * 8 + 4]);
        const float4 pp = *reinterpret_cast<const float4*>(&Ps[k][tx * 4]);
        const float2 x[4] = {make_float2(xa.x, xa.y), make_float2(xa.z, xa.w),
                             make_float2(xb.x, xb.y), make_float2(xb.z, xb.w)};
        const float p[4] = {pp.x, pp.y, pp.z, pp.w};
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
          for (int i = 0; i < 4; ++i)
            acc[i][t] = __ffma2_rn(x[i], make_float2(p[t], p[t]), acc[i][t]);
      };
      step(kk, aE);
      step(kk + 1, aO);
    }
  }
  float accE[8][4], accO[8][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      accE[2 * i][t] = aE[i][t].x;
      accE[2 * i + 1][t] = aE[i][t].y;
      accO[2 * i][t] = aO[i][t].x;
      accO[2 * i + 1][t] = aO[i][t].y;
    }

#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int r = r0 + ty * 8 + i;
    if (r >= rows) continue;
    int b, row;
    row_map(m, r, b, row);
    float* o = out + ((size_t)b * M + row) * J;
    const int jv = j0 + tx * 4;
    if ((J & 3) == 0 && jv + 3 < Jh) {
      // Row starts are 16-byte aligned; the mirrored block J-4-jv.. is too.
      *reinterpret_cast<float4*>(o + jv) =
          make_float4(accE[i][0] + accO[i][0], accE[i][1] + accO[i][1],
                      accE[i][2] + accO[i][2], accE[i][3] + accO[i][3]);
      *reinterpret_cast<float4*>(o + (J - 4 - jv)) =
          make_float4(accE[i][3] - accO[i][3], accE[i][2] - accO[i][2],
                      accE[i][1] - accO[i][1], accE[i][0] - accO[i][0]);
      continue;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      int j = jv + t;
      if (j >= Jh) continue;
      o[j] = accE[i][t] + accO[i][t];
      int jm = J - 1 - j;
      if (jm != j) o[jm] = accE[i][t] - accO[i][t];
    }
  }
}

// out_modal[b][row][l] = sum_j p[m,j,l] G[b][row][j] (forward contraction);
// writes zeros for l < m.  A CTA covers TB rows and TN values of l (64 for
// long l ranges, 32 for short ones, which keeps more CTAs per SM): thread
// (tx, ty) accumulates rows 8 ty .. 8 ty + 7 at l - m = k0 + tx + 8 t,
// t < TN / 8, all of one parity, so it reads only the symmetric (even) or
// antisymmetric (odd) latitude fold.  Folds and table chunks are fetched with
// float4 loads where the rows allow.
// Two rows share an f32x2 FMA, and the two folds lie half a bank line apart,
// because the lanes of a read take both: TL159, 75 fields 44.4 -> 36.7 us, T42,
// 900 fields 17.9 -> 15.3, TL255, 64 fields 74.3 -> 68.3, TL95, 600 fields 51.0 ->
// 47.6.
template <int TN, int TB>
__global__ void __launch_bounds__(TB)
legendre_forward_simt(const float* G, float* __restrict__ out,
                      int B, int M, int L, int J, int Jh,
                      const float* __restrict__ ptab,
                      const int64_t* __restrict__ ptab_off) {
  pdl_trigger();
  pdl_wait();
  const int m = blockIdx.z;
  const int rows = (m == 0) ? B : 2 * B;
  const int r0 = blockIdx.y * TB;
  if (r0 >= rows) return;
  const int Lm = L - m;
  constexpr int TT = TN / 8;           // l values per thread
  constexpr int PV = TN * kLegKC / TB; // table values fetched per thread and chunk
  constexpr int PT = kLegKC / PV;      // threads per table row
  const int k0 = blockIdx.x * TN;  // l - m offset of this tile
  const int tid = threadIdx.x;
  const int tx = tid & 7;
  const int ty = tid >> 3;

  if (blockIdx.x == 0 && m > 0) {
    // Structural zeros l < m of the rows handled by this CTA.
    for (int idx = tid; idx < TB * m; idx += TB) {
      int rl = idx / m, l = idx % m;
      int r = r0 + rl;
      if (r < rows) {
        int b, row;
        row_map(m, r, b, row);
        out[((size_t)b * M + row) * L + l] = 0.f;
      }
    }
  }
  if (k0 >= Lm) return;
  const float* P = ptab + ptab_off[m];

  // The antisymmetric fold lies half a bank line (16 floats) off the symmetric
  // one's banks: the lanes of a read take both.
  constexpr int kFoldStride = TB + 4, kDs = kLegKC * kFoldStride + 16;
  __shared__ __align__(16) float folds[kDs + kLegKC * kFoldStride];
  float(*Ss)[kFoldStride] = reinterpret_cast<float(*)[kFoldStride]>(folds);
  float(*Ds)[kFoldStride] = reinterpret_cast<float(*)[kFoldStride]>(folds + kDs);
  __shared__ float Ps[kLegKC][TN + 1];

  const int lq = tid & 3;
  const float* grow[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + (tid >> 2) + TB / 4 * i;
    grow[i] = nullptr;
    if (r < rows) {
      int b, row;
      row_map(m, r, b, row);
      grow[i] = G + ((size_t)b * M + row) * J;
    }
  }
  // Row starts are 16-byte aligned when J % 4 == 0 (then so are j and the
  // mirrored J - 4 - j for j a multiple of 4).
  const bool vec = (J & 3) == 0;
  // P chunk TN (l) x 16 (j): thread loads l = tid / PT, j = PV (tid % PT) ..
  const int pl_ = tid / PT, pjq = (tid % PT) * PV;
  float sv[4][4], dv[4][4], pvr[PV];
  auto fetch = [&](int jc) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = jc + lq * 4;
      float g1[4] = {0.f, 0.f, 0.f, 0.f}, g2[4] = {0.f, 0.f, 0.f, 0.f};
      if (grow[i]) {
        if (vec && j + 4 <= Jh) {
          const float4 d = *reinterpret_cast<const float4*>(grow[i] + j);
          const float4 e = *reinterpret_cast<const float4*>(grow[i] + J - 4 - j);
          g1[0] = d.x; g1[1] = d.y; g1[2] = d.z; g1[3] = d.w;
          g2[0] = e.w; g2[1] = e.z; g2[2] = e.y; g2[3] = e.x;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (j + e < Jh) {
              g1[e] = grow[i][j + e];
              const int jm = J - 1 - (j + e);
              g2[e] = (jm != j + e) ? grow[i][jm] : 0.f;
            }
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sv[i][e] = g1[e] + g2[e];
        dv[i][e] = g1[e] - g2[e];
      }
    }
    const int k = k0 + pl_;
    const int j = jc + pjq;
    const float* pr = P + (size_t)k * Jh + j;
    if ((Jh & 3) == 0 && k < Lm && j + PV <= Jh) {
      // Table rows start 16-byte aligned (the per-m offsets are multiples of
      // Jh).
#pragma unroll
      for (int q = 0; q < PV / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(pr + 4 * q);
        pvr[4 * q] = v.x;
        pvr[4 * q + 1] = v.y;
        pvr[4 * q + 2] = v.z;
        pvr[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int e = 0; e < PV; ++e) pvr[e] = (k < Lm && j + e < Jh) ? pr[e] : 0.f;
    }
  };

  float2 acc[4][TT];  // row pairs
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[i][t] = make_float2(0.f, 0.f);

  fetch(0);
  for (int jc = 0; jc < Jh; jc += kLegKC) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        Ss[lq * 4 + e][(tid >> 2) + TB / 4 * i] = sv[i][e];
        Ds[lq * 4 + e][(tid >> 2) + TB / 4 * i] = dv[i][e];
      }
#pragma unroll
    for (int e = 0; e < PV; ++e) Ps[pjq + e][pl_] = pvr[e];
    __syncthreads();
    if (jc + kLegKC < Jh) fetch(jc + kLegKC);
    const float* fold = (tx & 1) ? &Ds[0][0] : &Ss[0][0];
#pragma unroll
    for (int jj = 0; jj < kLegKC; ++jj) {
      float4 fa = *reinterpret_cast<const float4*>(fold + jj * (TB + 4) + ty * 8);
      float4 fb = *reinterpret_cast<const float4*>(fold + jj * (TB + 4) + ty * 8 + 4);
      const float2 f4[4] = {make_float2(fa.x, fa.y), make_float2(fa.z, fa.w),
                            make_float2(fb.x, fb.y), make_float2(fb.z, fb.w)};
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const float pw = Ps[jj][tx + 8 * t];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          acc[i][t] = __ffma2_rn(f4[i], make_float2(pw, pw), acc[i][t]);
      }
    }
  }

#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int r = r0 + ty * 8 + i;
    if (r >= rows) continue;
    int b, row;
    row_map(m, r, b, row);
    float* o = out + ((size_t)b * M + row) * L + m;
#pragma unroll
    for (int t = 0; t < TT; ++t) {
      int k = k0 + tx + 8 * t;
      if (k < Lm) o[k] = (i & 1) ? acc[i >> 1][t].y : acc[i >> 1][t].x;
    }
  }
}

// Rows per CTA: 64 where that saves half a row tile of one or two (rows of one
// or three 64-row tiles), or where 128 leave fewer than `few` CTAs; else 128,
// which reads the table half as often.  Forward / inverse us with 128 and 64
// rows: T213, 20 fields (40 rows) 55.9 -> 42.1 / 30.2 -> 24.2; T85, 15 fields 16.6
// -> 14.6; TL159, 75 fields (150 rows) 36.9, 37.0 / 24.8 -> 21.8; T42, 121 fields
// (172 CTAs forward) 9.6 -> 8.1; TL127, 33 fields inverse 12.7 -> 14.2; TL255, 64
// fields 68 -> 74.
static int leg_rows(const dino_plan* p, int nf, int tiles, int few) {
  const int half = ceil_div(2 * nf, 64);
  const bool short_grid = (int64_t)ceil_div(2 * nf, 128) * tiles * p->lw < few;
  return (half == 1 || half == 3 || short_grid) ? 64 : 128;
}

// The FP32 SIMT inverse contraction regardless of the plan's precision.
int legendre_inverse_fp32(dino_plan* p, const Segs& in, float* out, int nf,
                          cudaStream_t st) {
  NvtxRange range("inv_legendre");
  const int tiles = ceil_div(p->Jh, kLegTN), tb = leg_rows(p, nf, tiles, 0);
  return launch_pdl("legendre_inverse_simt",
                    tb == 64 ? legendre_inverse_simt<64> : legendre_inverse_simt<128>,
                    dim3(tiles, ceil_div(2 * nf, tb), p->lw), tb, 0, st, in, out, nf, p->M, p->L,
                    p->J, p->Jh, p->d_ptab, p->d_ptab_off);
}

int legendre_inverse(dino_plan* p, const Segs& in, float* out, int nf,
                     cudaStream_t st) {
  if (p->precision != DINO_PREC_FP32 && !tc_use_simt(p, false)) {
    NvtxRange range("inv_legendre");
    return tc_legendre_inverse(p, in, out, nf, st);
  }
  return legendre_inverse_fp32(p, in, out, nf, st);
}

int legendre_forward(dino_plan* p, const float* G, float* out, int nf,
                     cudaStream_t st) {
  NvtxRange range("fwd_legendre");
  if (p->precision != DINO_PREC_FP32 && !tc_use_simt(p, true))
    return tc_legendre_forward(p, G, out, nf, st);
  return legendre_forward_fp32(p, G, out, nf, st);
}

// The FP32 SIMT forward contraction regardless of the plan's precision.
int legendre_forward_fp32(dino_plan* p, const float* G, float* out, int nf,
                          cudaStream_t st) {
  const int tn = p->L > 64 ? 64 : 32, tiles = ceil_div(p->L, tn);
  const int tb = leg_rows(p, nf, tiles, 2 * p->sms);
  auto* kernel = tn == 64
                     ? (tb == 64 ? legendre_forward_simt<64, 64> : legendre_forward_simt<64, 128>)
                     : (tb == 64 ? legendre_forward_simt<32, 64> : legendre_forward_simt<32, 128>);
  return launch_pdl("legendre_forward_simt", kernel, dim3(tiles, ceil_div(2 * nf, tb), p->lw), tb,
                    0, st, G, out, nf, p->M, p->L, p->J, p->Jh, p->d_ptab, p->d_ptab_off);
}

// ---------------------------------------------------------------------------
// Real FFT over longitude (I = 2N, N of FftCfg below): shared-memory Stockham
// passes on the half-length complex sequence z[n] = x[2n] + i x[2n+1].
//
// A thread works on two adjacent latitudes at once, so every complex value is
// a pair of packed f32x2 registers (re of both columns, im of both columns):
// one issue slot does both columns' add, multiply or FMA at the plain lane
// rate (126 lane results per SM and clock, measured for fma and fma.f32x2
// alike).  With one column per thread the kernels issued in 57-70 % of the
// slots; now 29-34 %, and they wait on memory (long scoreboard is the largest
// stall at TL255).  T42 x 900 fields: inverse 18.6 -> 12.4 us, forward 14.7 ->
// 10.6 us; T85 x 128: 10.7 -> 8.4, 10.5 -> 8.4 us; TL255 x 128: 37.0 -> 32.2,
// 33.0 -> 29.7 us (with launches overlapping).  Against direct sums for lengths that are no power of two:
// TL159 x 75 fields 615 -> 10.4 us and 636 -> 10.4 us.
// ---------------------------------------------------------------------------

// Packed arithmetic on two columns.
__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) {
  return __ffma2_rn(a, b, c);
}
// a - b (one rounding: b * -1 is exact).
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
  return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// One complex value of two columns.
struct cpair {
  float2 re, im;
};
__device__ __forceinline__ cpair cadd(cpair a, cpair b) {
  return {padd(a.re, b.re), padd(a.im, b.im)};
}
__device__ __forceinline__ cpair csub(cpair a, cpair b) {
  return {psub(a.re, b.re), psub(a.im, b.im)};
}
// a + i kSign b and a - i kSign b: a quarter turn is a choice of operands.
template <int kSign>
__device__ __forceinline__ cpair cadd_i(cpair a, cpair b) {
  return kSign > 0 ? cpair{psub(a.re, b.im), padd(a.im, b.re)}
                   : cpair{padd(a.re, b.im), psub(a.im, b.re)};
}
template <int kSign>
__device__ __forceinline__ cpair csub_i(cpair a, cpair b) {
  return cadd_i<-kSign>(a, b);
}
// a (wr + i wi), the same factor for both columns; nwi = -wi.  One product of
// each part is rounded, the other is inside the FMA.
__device__ __forceinline__ cpair cmul_w(cpair a, float2 wr, float2 wi, float2 nwi) {
  return {pfma(a.re, wr, pmul(a.im, nwi)), pfma(a.re, wi, pmul(a.im, wr))};
}

// Multiplies by exp(kSign 2 pi i K / 16) for a compile-time K in [0, 9].
template <int K, int kSign>
__device__ __forceinline__ cpair twiddle16(cpair a) {
  constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f;
  constexpr float h = 0.70710678118654757f;
  constexpr float co[10] = {1.f, c1, h, s1, 0.f, -s1, -h, -c1, -1.f, -c1};
  constexpr float si[10] = {0.f, s1, h, c1, 1.f, c1, h, s1, 0.f, -s1};
  if constexpr (K == 0) {
    return a;
  } else if constexpr (K == 4) {
    const float2 z = make_float2(0.f, 0.f);
    return kSign > 0 ? cpair{psub(z, a.im), a.re} : cpair{a.im, psub(z, a.re)};
  } else {
    constexpr float wi = kSign * si[K];
    return cmul_w(a, dup(co[K]), dup(wi), dup(-wi));
  }
}

// DFT of length 4: X_k = sum_q v_q exp(kSign 2 pi i q k / 4).
template <int kSign>
__device__ __forceinline__ void dft4(cpair& a, cpair& b, cpair& c, cpair& d) {
  const cpair s0 = cadd(a, c), d0 = csub(a, c);
  const cpair s1 = cadd(b, d), d1 = csub(b, d);
  a = cadd(s0, s1);
  c = csub(s0, s1);
  b = cadd_i<kSign>(d0, d1);
  d = csub_i<kSign>(d0, d1);
}

template <int R, int kSign>
__device__ __forceinline__ void dft_reg(cpair* v);

// In-register DFT of length A B with A and B coprime (Good 1958; Thomas
// 1963): the inputs n = B n1 + A n2 (mod A B) make it an A x B
// two-dimensional DFT without twiddles, whose entry (k mod A, k mod B) is X_k.
template <int A, int B, int kSign>
__device__ __forceinline__ void dft_coprime(cpair* v) {
  constexpr int R = A * B;
  cpair t[R];
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1) {
    cpair row[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) row[n2] = v[(B * n1 + A * n2) % R];
    dft_reg<B, kSign>(row);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) t[n1 * B + k2] = row[k2];
  }
#pragma unroll
  for (int k2 = 0; k2 < B; ++k2) {
    cpair col[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) col[n1] = t[n1 * B + k2];
    dft_reg<A, kSign>(col);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) t[k1 * B + k2] = col[k1];
  }
#pragma unroll
  for (int k = 0; k < R; ++k) v[k] = t[(k % A) * B + k % B];
}

// In-register DFT of length R, natural order in and out:
// v_s <- sum_q v_q exp(kSign 2 pi i q s / R).
template <int R, int kSign>
__device__ __forceinline__ void dft_reg(cpair* v) {
  if constexpr (R == 2) {
    const cpair a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 3) {
    // X1,2 = (a - (b + c) / 2) +- i sin(pi/3) (b - c).
    constexpr float s3 = 0.86602540378443865f;
    const cpair t = cadd(v[1], v[2]), u = csub(v[1], v[2]);
    const cpair m = {pfma(t.re, dup(-0.5f), v[0].re), pfma(t.im, dup(-0.5f), v[0].im)};
    const float2 p = dup(kSign * s3), n = dup(-kSign * s3);
    v[0] = cadd(v[0], t);
    v[1] = {pfma(u.im, n, m.re), pfma(u.re, p, m.im)};
    v[2] = {pfma(u.im, p, m.re), pfma(u.re, n, m.im)};
  } else if constexpr (R == 4) {
    dft4<kSign>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 5) {
    constexpr float c1 = 0.30901699437494742f, c2 = -0.80901699437494742f;
    constexpr float s1 = 0.95105651629515357f, s2 = 0.58778525229247313f;
    const cpair t1 = cadd(v[1], v[4]), u1 = csub(v[1], v[4]);
    const cpair t2 = cadd(v[2], v[3]), u2 = csub(v[2], v[3]);
    const cpair m1 = {pfma(t2.re, dup(c2), pfma(t1.re, dup(c1), v[0].re)),
                      pfma(t2.im, dup(c2), pfma(t1.im, dup(c1), v[0].im))};
    const cpair m2 = {pfma(t2.re, dup(c1), pfma(t1.re, dup(c2), v[0].re)),
                      pfma(t2.im, dup(c1), pfma(t1.im, dup(c2), v[0].im))};
    const cpair w1 = {pfma(u2.re, dup(s2), pmul(u1.re, dup(s1))),
                      pfma(u2.im, dup(s2), pmul(u1.im, dup(s1)))};
    const cpair w2 = {pfma(u2.re, dup(-s1), pmul(u1.re, dup(s2))),
                      pfma(u2.im, dup(-s1), pmul(u1.im, dup(s2)))};
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd_i<kSign>(m1, w1);
    v[4] = csub_i<kSign>(m1, w1);
    v[2] = cadd_i<kSign>(m2, w2);
    v[3] = csub_i<kSign>(m2, w2);
  } else if constexpr (R == 8) {
    cpair e[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      e[i] = v[2 * i];
      o[i] = v[2 * i + 1];
    }
    dft_reg<4, kSign>(e);
    dft_reg<4, kSign>(o);
    o[1] = twiddle16<2, kSign>(o[1]);
    o[3] = twiddle16<6, kSign>(o[3]);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], o[1]);
    v[5] = csub(e[1], o[1]);
    v[2] = cadd_i<kSign>(e[2], o[2]);
    v[6] = csub_i<kSign>(e[2], o[2]);
    v[3] = cadd(e[3], o[3]);
    v[7] = csub(e[3], o[3]);
  } else if constexpr (R == 16) {
    // q = 4 q1 + q2, s = s1 + 4 s2: DFT-4 over q1 for each q2, twiddle
    // W16^(q2 s1), DFT-4 over q2 for each s1.
    cpair y[16];
#pragma unroll
    for (int q2 = 0; q2 < 4; ++q2) {
      cpair a = v[q2], b = v[4 + q2], c = v[8 + q2], d = v[12 + q2];
      dft4<kSign>(a, b, c, d);
      y[4 * q2] = a;
      y[4 * q2 + 1] = b;
      y[4 * q2 + 2] = c;
      y[4 * q2 + 3] = d;
    }
    y[5] = twiddle16<1, kSign>(y[5]);
    y[6] = twiddle16<2, kSign>(y[6]);
    y[7] = twiddle16<3, kSign>(y[7]);
    y[9] = twiddle16<2, kSign>(y[9]);
    y[10] = twiddle16<4, kSign>(y[10]);
    y[11] = twiddle16<6, kSign>(y[11]);
    y[13] = twiddle16<3, kSign>(y[13]);
    y[14] = twiddle16<6, kSign>(y[14]);
    y[15] = twiddle16<9, kSign>(y[15]);
#pragma unroll
    for (int s1 = 0; s1 < 4; ++s1) {
      cpair a = y[s1], b = y[4 + s1], c = y[8 + s1], d = y[12 + s1];
      dft4<kSign>(a, b, c, d);
      v[s1] = a;
      v[s1 + 4] = b;
      v[s1 + 8] = c;
      v[s1 + 12] = d;
    }
  } else if constexpr (R == 6) {
    dft_coprime<2, 3, kSign>(v);
  } else if constexpr (R == 10) {
    dft_coprime<2, 5, kSign>(v);
  } else if constexpr (R == 12) {
    dft_coprime<3, 4, kSign>(v);
  } else if constexpr (R == 15) {
    dft_coprime<3, 5, kSign>(v);
  } else {
    static_assert(R == 20, "radix");
    dft_coprime<4, 5, kSign>(v);
  }
}

// Radices (at most three passes), threads, the CTAs per SM that bound the
// registers, and column pairs per CTA for each supported half length: every N
// of the named grids.  Passes are few and wide (a pass costs a round trip
// through shared memory and a barrier) and the thread count is near the widest
// pass's N / R x pairs items.  16 pairs make a row segment a full 128-byte
// line: TL255 (N = 256), 128 fields: 2 CTAs of 256 threads and 16 pairs 37.1 /
// 31.1 us (inverse / forward), pair 146 us; 5 of 128 threads and 8 pairs 37.2 /
// 35.0 us, 155 us; a register bound of 80 (6 CTAs) 43 / 45 us.  T42 (N = 64),
// 900 fields: 16 pairs 12.4 / 10.6 us, 8 pairs 12.6 / 12.6 us.  Shorter rows
// (N <= 48) and the lengths whose passes hold 60-80 registers (160 on) keep 8.
template <int N> struct FftCfg;
#define DINO_FFT_CFG(N, R1, R2, R3, THREADS, CTAS, PAIRS)                  \
  template <> struct FftCfg<N> {                                           \
    static constexpr int r1 = R1, r2 = R2, r3 = R3, threads = THREADS,     \
                         ctas = CTAS, pairs = PAIRS;                       \
    static_assert(R1 * R2 * R3 == N && THREADS % PAIRS == 0, "radices");    \
  };
DINO_FFT_CFG(8, 8, 1, 1, 32, 16, 8)
DINO_FFT_CFG(16, 16, 1, 1, 32, 16, 8)
DINO_FFT_CFG(32, 8, 4, 1, 64, 14, 8)
DINO_FFT_CFG(48, 8, 6, 1, 64, 14, 8)
DINO_FFT_CFG(64, 8, 8, 1, 128, 5, 16)
DINO_FFT_CFG(96, 12, 8, 1, 192, 4, 16)
DINO_FFT_CFG(128, 16, 8, 1, 128, 4, 16)
DINO_FFT_CFG(160, 16, 10, 1, 128, 5, 8)
DINO_FFT_CFG(180, 12, 15, 1, 128, 5, 8)
DINO_FFT_CFG(256, 16, 16, 1, 256, 2, 16)
DINO_FFT_CFG(320, 16, 20, 1, 160, 3, 8)
DINO_FFT_CFG(512, 8, 8, 8, 256, 2, 8)
DINO_FFT_CFG(640, 8, 8, 10, 320, 2, 8)
DINO_FFT_CFG(1280, 16, 8, 10, 640, 1, 8)
#undef DINO_FFT_CFG

bool fft_supported(int n) {
  switch (n) {
    case 8: case 16: case 32: case 48: case 64: case 96: case 128: case 160:
    case 180: case 256: case 320: case 512: case 640: case 1280:
      return true;
  }
  return false;
}

// Shared memory of both kernels: N x pairs complex column pairs and the N
// twiddles exp(kSign 2 pi i k / N) as (re, re, im, im).
template <int N>
constexpr size_t fft_smem_bytes() {
  return sizeof(float4) * ((size_t)N * FftCfg<N>::pairs + N);
}

__device__ __forceinline__ cpair ld_cpair(const float4* s) {
  const float4 t = *s;
  return {make_float2(t.x, t.y), make_float2(t.z, t.w)};
}
__device__ __forceinline__ void st_cpair(float4* s, cpair v) {
  *s = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}

// One radix-R Stockham pass over N points for P column pairs.
// load(n) returns element n of the thread's column pair (tid mod P in
// every pass); store(n, v) writes output element n.  Every thread issues all
// of its loads before its first store; kSync puts a barrier between the two,
// so that the pass may run in place on one shared buffer.
template <int N, int R, int Ns, int kSign, bool kSync, class Load, class Store>
__device__ __forceinline__ void stockham_pass(const float4* tw, Load load, Store store) {
  constexpr int T = FftCfg<N>::threads;
  constexpr int Q = N / R;
  constexpr int P = FftCfg<N>::pairs;
  constexpr int kRows = T / P;  // items per column pair and round
  constexpr int kItems = (Q + kRows - 1) / kRows;
  constexpr int stride = N / (Ns * R);
  const int j0 = threadIdx.x / P;
  cpair v[kItems][R];
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int j = j0 + it * kRows;
    if (j < Q) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[it][r] = load(j + r * Q);
    }
  }
  if (kSync) __syncthreads();
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int j = j0 + it * kRows;
    if (j < Q) {
      const int k = j % Ns;
      if constexpr (Ns > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r) {
          const float4 w = tw[r * k * stride];
          const float2 wr = make_float2(w.x, w.y), wi = make_float2(w.z, w.w);
          v[it][r] = cmul_w(v[it][r], wr, wi, pmul(wi, dup(-1.f)));
        }
      }
      dft_reg<R, kSign>(v[it]);
      const int base = (j / Ns) * Ns * R + k;
#pragma unroll
      for (int r = 0; r < R; ++r) store(base + r * Ns, v[it][r]);
    }
  }
}

// Runs all passes; the first reads via `first` (in place on S when kFirstInS)
// and the last writes via `last` (in place on S when kLastInS).
template <int N, int kSign, bool kFirstInS, bool kLastInS, class First, class Last>
__device__ __forceinline__ void fft_passes(float4* S, const float4* tw, First first,
                                           Last last) {
  using C = FftCfg<N>;
  constexpr int P = C::pairs;
  const int p = threadIdx.x % P;
  auto s_load = [S, p](int n) { return ld_cpair(S + n * P + p); };
  auto s_store = [S, p](int n, cpair v) { st_cpair(S + n * P + p, v); };
  if constexpr (C::r2 == 1) {
    stockham_pass<N, C::r1, 1, kSign, kFirstInS && kLastInS>(tw, first, last);
  } else if constexpr (C::r3 == 1) {
    stockham_pass<N, C::r1, 1, kSign, kFirstInS>(tw, first, s_store);
    __syncthreads();
    stockham_pass<N, C::r2, C::r1, kSign, kLastInS>(tw, s_load, last);
  } else {
    stockham_pass<N, C::r1, 1, kSign, kFirstInS>(tw, first, s_store);
    __syncthreads();
    stockham_pass<N, C::r2, C::r1, kSign, true>(tw, s_load, s_store);
    __syncthreads();
    stockham_pass<N, C::r3, C::r1 * C::r2, kSign, kLastInS>(tw, s_load, last);
  }
}

// The two columns of a row for one thread: one 8-byte access when kVec (even
// J and 8-byte aligned bases, so `cols` is 0 or 2), else scalar ones.
template <bool kVec>
__device__ __forceinline__ float2 ld_cols(const float* g, int cols) {
  if (kVec)
    return cols ? *reinterpret_cast<const float2*>(g) : make_float2(0.f, 0.f);
  return make_float2(cols > 0 ? g[0] : 0.f, cols > 1 ? g[1] : 0.f);
}
template <bool kVec>
__device__ __forceinline__ void st_cols(float* g, float2 v, int cols) {
  if (kVec) {
    if (cols) *reinterpret_cast<float2*>(g) = v;
  } else {
    if (cols > 0) g[0] = v.x;
    if (cols > 1) g[1] = v.y;
  }
}

// Fourier coefficients F[b][row][j] -> nodal[b][i][j] (optionally scaled by
// wq[j], which gives the adjoint of the weighted forward transform).
// With A = X[k] + conj X[N-k], B = X[k] - conj X[N-k] and T = w_I^k B, the
// half-length spectrum is Z[k] = A + i T and Z[N-k] = conj(A) + i conj(T)
// (w_I^(N-k) = -conj w_I^k); then z = IDFT_N(Z) and x[2n] = Re z[n],
// x[2n+1] = Im z[n].  Z is formed from the coefficients' global rows (four
// 8-byte loads an item, eight items in flight a thread), the first passes run
// in place in shared memory and the last writes the nodal rows.
template <int N, bool kVec>
__global__ void __launch_bounds__(FftCfg<N>::threads, FftCfg<N>::ctas)
rfft_inverse_kernel(const float* F, float* __restrict__ out,
                    int M, int lw, int J, const float2* __restrict__ tw_n,
                    const float2* __restrict__ tw_i,
                    const float* __restrict__ wq) {
  pdl_trigger();
  constexpr int T = FftCfg<N>::threads, P = FftCfg<N>::pairs;
  extern __shared__ float4 sm[];
  float4* S = sm;
  float4* tw = S + N * P;
  const int tid = threadIdx.x, p = tid % P;
  const int b = blockIdx.y;
  const int col = (blockIdx.x * P + p) * 2;
  const int cols = max(0, min(2, J - col));
  for (int t = tid; t < N; t += T) {
    const float2 w = tw_n[t];
    tw[t] = make_float4(w.x, w.x, w.y, w.y);
  }
  pdl_wait();
  const float* Fb = F + (size_t)b * M * J + col;
  const float inv_sqrt_2pi = 0.3989422804014327f;
  const float half_inv_sqrt_pi = 0.28209479177387814f;
  const float2 wc = wq ? ld_cols<false>(wq + col, cols) : make_float2(1.f, 1.f);
  const float2 sc = pmul(wc, dup(half_inv_sqrt_pi));
  // Items k = 0 .. N/2 - 1: the pair (k, N - k), and for k = 0 the two terms
  // without a partner, Z[0] and Z[N/2].
  constexpr int kRows = T / P;
  constexpr int kAll = (N / 2 + kRows - 1) / kRows;
  constexpr int kBatch = kAll < 8 ? kAll : 8;
  const int k0 = tid / P;
#pragma unroll
  for (int i0 = 0; i0 < kAll; i0 += kBatch) {
    float2 ck[kBatch], sk[kBatch], cn[kBatch], sn[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int k = k0 + (i0 + i) * kRows;
      const int kn = k == 0 ? N / 2 : N - k;
      const int nk = (k < N / 2 && k < lw) ? cols : 0;
      const int nn = (k < N / 2 && kn < lw) ? cols : 0;
      const float* fk = Fb + (size_t)(k == 0 ? 0 : 2 * k - 1) * J;
      const float* fn = Fb + (size_t)(2 * kn - 1) * J;
      ck[i] = ld_cols<kVec>(fk, nk);
      sk[i] = ld_cols<kVec>(fk + J, k == 0 ? 0 : nk);
      cn[i] = ld_cols<kVec>(fn, nn);
      sn[i] = ld_cols<kVec>(fn + J, nn);
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const int k = k0 + (i0 + i) * kRows;
      if (k >= N / 2) continue;
      if (k == 0) {
        const float2 x0 = pmul(ck[i], pmul(wc, dup(inv_sqrt_2pi)));
        st_cpair(S + p, {x0, x0});
        const float2 two = padd(sc, sc);
        st_cpair(S + (N / 2) * P + p, {pmul(cn[i], two), pmul(sn[i], two)});
        continue;
      }
      const float2 a = pmul(ck[i], sc), s = pmul(sk[i], sc);
      const float2 c = pmul(cn[i], sc), d = pmul(sn[i], sc);
      const float2 ar = padd(a, c), ai = psub(d, s);
      const float2 br = psub(a, c), q = padd(s, d);  // B = br - i q
      const float2 w = tw_i[k];
      const float2 wr = dup(w.x), wi = dup(w.y);
      const float2 tr = pfma(br, wr, pmul(q, wi));
      const float2 ti = pfma(br, wi, pmul(q, dup(-w.x)));
      st_cpair(S + k * P + p, {psub(ar, ti), padd(ai, tr)});
      st_cpair(S + (N - k) * P + p, {padd(ar, ti), psub(tr, ai)});
    }
  }
  __syncthreads();
  float* ob = out + (size_t)b * (2 * N) * J + col;
  auto first = [S, p](int n) { return ld_cpair(S + n * P + p); };
  auto last = [ob, J, cols](int n, cpair v) {
    float* o = ob + (size_t)(2 * n) * J;
    st_cols<kVec>(o, v.re, cols);
    st_cols<kVec>(o + J, v.im, cols);
  };
  fft_passes<N, 1, true, false>(S, tw, first, last);
}

// nodal[b][i][j] -> F[b][row][j] (times wq[j] when given: the forward SHT's
// quadrature weights; without: the adjoint of the inverse transform).  The
// first pass reads the nodal rows, the last leaves Z in shared memory; with
// s = (Z[k] + conj Z[N-k]) / 2, d = (Z[k] - conj Z[N-k]) / 2 and
// U = -i conj(w_I^k) d, X[k] = s + U and X[N-k] = conj(s - U).
template <int N, bool kVec>
__global__ void __launch_bounds__(FftCfg<N>::threads, FftCfg<N>::ctas)
rfft_forward_kernel(const float* x, float* __restrict__ F, int M,
                    int lw, int J, const float2* __restrict__ tw_n,
                    const float2* __restrict__ tw_i,
                    const float* __restrict__ wq) {
  pdl_trigger();
  constexpr int T = FftCfg<N>::threads, P = FftCfg<N>::pairs;
  extern __shared__ float4 sm[];
  float4* S = sm;
  float4* tw = S + N * P;
  const int tid = threadIdx.x, p = tid % P;
  const int b = blockIdx.y;
  const int col = (blockIdx.x * P + p) * 2;
  const int cols = max(0, min(2, J - col));
  for (int t = tid; t < N; t += T) {
    const float2 w = tw_n[t];
    tw[t] = make_float4(w.x, w.x, -w.y, -w.y);
  }
  pdl_wait();
  const float* xb = x + (size_t)b * (2 * N) * J + col;
  auto first = [xb, J, cols](int n) -> cpair {
    const float* g = xb + (size_t)(2 * n) * J;
    return {ld_cols<kVec>(g, cols), ld_cols<kVec>(g + J, cols)};
  };
  auto last = [S, p](int n, cpair v) { st_cpair(S + n * P + p, v); };
  fft_passes<N, -1, false, true>(S, tw, first, last);
  __syncthreads();
  if (cols == 0) return;
  float* Fb = F + (size_t)b * M * J + col;
  const float inv_sqrt_2pi = 0.3989422804014327f;
  const float inv_sqrt_pi = 0.5641895835477563f;
  const float2 wc = wq ? ld_cols<false>(wq + col, cols) : make_float2(1.f, 1.f);
  const float2 a0 = pmul(wc, dup(inv_sqrt_2pi)), a1 = pmul(wc, dup(inv_sqrt_pi));
  const float2 ah = pmul(a1, dup(0.5f));
  constexpr int kRows = T / P;
#pragma unroll 4
  for (int k = tid / P; k < N / 2; k += kRows) {
    const int kn = k == 0 ? N / 2 : N - k;
    const cpair zk = ld_cpair(S + k * P + p);
    const cpair zn = ld_cpair(S + kn * P + p);
    float* fk = Fb + (size_t)(k == 0 ? 0 : 2 * k - 1) * J;
    float* fn = Fb + (size_t)(2 * kn - 1) * J;
    if (k == 0) {
      st_cols<kVec>(fk, pmul(padd(zk.re, zk.im), a0), cols);
      if (kn < lw) {
        st_cols<kVec>(fn, pmul(zn.re, a1), cols);
        st_cols<kVec>(fn + J, pmul(zn.im, a1), cols);
      }
      continue;
    }
    const float2 w = tw_i[k];
    const float2 wr = dup(w.x), wi = dup(w.y);
    const float2 sr = padd(zk.re, zn.re), si = psub(zk.im, zn.im);  // 2 s
    const float2 dr = psub(zk.re, zn.re), di = padd(zk.im, zn.im);  // 2 d
    const float2 ur = pfma(wr, di, pmul(dup(-w.y), dr));
    const float2 v = pfma(wi, di, pmul(wr, dr));  // -Im 2U
    if (k < lw) {
      st_cols<kVec>(fk, pmul(padd(sr, ur), ah), cols);
      st_cols<kVec>(fk + J, pmul(psub(v, si), ah), cols);
    }
    if (kn < lw) {
      st_cols<kVec>(fn, pmul(psub(sr, ur), ah), cols);
      st_cols<kVec>(fn + J, pmul(padd(si, v), ah), cols);
    }
  }
}

// Generic longitude transforms by direct summation with the FP32 real basis
// f[i][row] (any I, any lw <= I).
__global__ void dft_inverse_kernel(const float* F,
                                   float* __restrict__ out, int M, int I, int J,
                                   const float* __restrict__ f,
                                   const float* __restrict__ wq) {
  pdl_trigger();
  pdl_wait();
  int j = blockIdx.x * 32 + threadIdx.x;
  int i = blockIdx.y * 8 + threadIdx.y;
  int b = blockIdx.z;
  if (j >= J || i >= I) return;
  const float* Fb = F + (size_t)b * M * J + j;
  const float* fi = f + (size_t)i * M;
  float acc = 0.f;
  for (int r = 0; r < M; ++r) acc = fmaf(fi[r], Fb[(size_t)r * J], acc);
  if (wq) acc *= wq[j];
  out[((size_t)b * I + i) * J + j] = acc;
}

__global__ void dft_forward_kernel(const float* x,
                                   float* __restrict__ F, int M, int I, int J,
                                   const float* __restrict__ f,
                                   const float* __restrict__ wq) {
  pdl_trigger();
  pdl_wait();
  int j = blockIdx.x * 32 + threadIdx.x;
  int r = blockIdx.y * 8 + threadIdx.y;
  int b = blockIdx.z;
  if (j >= J || r >= M) return;
  const float* xb = x + (size_t)b * I * J + j;
  float acc = 0.f;
  for (int i = 0; i < I; ++i) acc = fmaf(f[(size_t)i * M + r], xb[(size_t)i * J], acc);
  if (wq) acc *= wq[j];
  F[((size_t)b * M + r) * J + j] = acc;
}

template <int N>
static int configure_rfft() {
  // Kernel attributes are set once per device, outside any stream capture
  // (sht_prepare runs this at plan creation on the plan's device).
  static PerDeviceOnce once;
  return once.run([] {
    const int smem = (int)fft_smem_bytes<N>();
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    DINO_CHECK_CUDA(cudaFuncSetAttribute(rfft_inverse_kernel<N, true>, attr, smem));
    DINO_CHECK_CUDA(cudaFuncSetAttribute(rfft_inverse_kernel<N, false>, attr, smem));
    DINO_CHECK_CUDA(cudaFuncSetAttribute(rfft_forward_kernel<N, true>, attr, smem));
    DINO_CHECK_CUDA(cudaFuncSetAttribute(rfft_forward_kernel<N, false>, attr, smem));
    return DINO_OK;
  });
}

template <int N>
static int launch_rfft(dino_plan* p, const float* in, float* out, int nf,
                       bool inverse, const float* wq, cudaStream_t st) {
  constexpr int T = FftCfg<N>::threads;
  const size_t smem = fft_smem_bytes<N>();
  if (!p) return configure_rfft<N>();
  DINO_TRY(configure_rfft<N>());
  dim3 grid(ceil_div(p->J, 2 * FftCfg<N>::pairs), nf);
  // Two columns per 8-byte access where every row starts 8-byte aligned.
  const bool vec = p->J % 2 == 0 && (reinterpret_cast<uintptr_t>(in) & 7) == 0 &&
                   (reinterpret_cast<uintptr_t>(out) & 7) == 0;
  auto* kernel = inverse ? (vec ? rfft_inverse_kernel<N, true> : rfft_inverse_kernel<N, false>)
                         : (vec ? rfft_forward_kernel<N, true> : rfft_forward_kernel<N, false>);
  return launch_pdl(inverse ? "rfft_inverse" : "rfft_forward", kernel, grid, T, smem, st, in, out,
                    p->M, p->lw, p->J, p->d_tw_n, p->d_tw_i, wq);
}

static int rfft_dispatch_n(int n, dino_plan* p, const float* in, float* out,
                           int nf, bool inverse, const float* wq,
                           cudaStream_t st) {
  switch (n) {
    case 8: return launch_rfft<8>(p, in, out, nf, inverse, wq, st);
    case 16: return launch_rfft<16>(p, in, out, nf, inverse, wq, st);
    case 32: return launch_rfft<32>(p, in, out, nf, inverse, wq, st);
    case 48: return launch_rfft<48>(p, in, out, nf, inverse, wq, st);
    case 64: return launch_rfft<64>(p, in, out, nf, inverse, wq, st);
    case 96: return launch_rfft<96>(p, in, out, nf, inverse, wq, st);
    case 128: return launch_rfft<128>(p, in, out, nf, inverse, wq, st);
    case 160: return launch_rfft<160>(p, in, out, nf, inverse, wq, st);
    case 180: return launch_rfft<180>(p, in, out, nf, inverse, wq, st);
    case 256: return launch_rfft<256>(p, in, out, nf, inverse, wq, st);
    case 320: return launch_rfft<320>(p, in, out, nf, inverse, wq, st);
    case 512: return launch_rfft<512>(p, in, out, nf, inverse, wq, st);
    case 640: return launch_rfft<640>(p, in, out, nf, inverse, wq, st);
    case 1280: return launch_rfft<1280>(p, in, out, nf, inverse, wq, st);
  }
  set_error("internal: unsupported FFT length");
  return DINO_ERR_UNSUPPORTED;
}

static int rfft_dispatch(dino_plan* p, const float* in, float* out, int nf,
                         bool inverse, const float* wq, cudaStream_t st) {
  return rfft_dispatch_n(p->N, p, in, out, nf, inverse, wq, st);
}

int sht_prepare(dino_plan* p) {
  if (!p->fft) return DINO_OK;
  return rfft_dispatch_n(p->N, nullptr, nullptr, nullptr, 0, true, nullptr, 0);
}

int fourier_inverse(dino_plan* p, const float* F, float* nodal, int nf,
                    bool weighted_adjoint, cudaStream_t st) {
  NvtxRange range("inv_fourier");
  const float* wq = weighted_adjoint ? p->d_wq : nullptr;
  if (p->fft) return rfft_dispatch(p, F, nodal, nf, true, wq, st);
  dim3 grid(ceil_div(p->J, 32), ceil_div(p->I, 8), nf);
  return launch_pdl("dft_inverse", dft_inverse_kernel, grid, dim3(32, 8), 0, st, F, nodal, p->M,
                    p->I, p->J, p->d_fbasis, wq);
}

int fourier_forward(dino_plan* p, const float* nodal, float* F, int nf,
                    bool weighted, cudaStream_t st) {
  NvtxRange range("fwd_fourier");
  const float* wq = weighted ? p->d_wq : nullptr;
  if (p->fft) return rfft_dispatch(p, nodal, F, nf, false, wq, st);
  dim3 grid(ceil_div(p->J, 32), ceil_div(p->M, 8), nf);
  return launch_pdl("dft_forward", dft_forward_kernel, grid, dim3(32, 8), 0, st, nodal, F, p->M,
                    p->I, p->J, p->d_fbasis, wq);
}

// ---------------------------------------------------------------------------
// Transform drivers (chunked by workspace capacity)
// ---------------------------------------------------------------------------

// Fields per launch such that the intermediate Fourier coefficients of one
// chunk (fields x M x J floats) stay resident in L2 between the Legendre and
// FFT kernels; chunks are balanced, and on the tensor-core path whole
// 128-row MMA tiles (64 fields) where the cap allows.
int l2_chunk(dino_plan* p, int nf, int work_fields) {
  const size_t per_field = (size_t)p->M * p->J * sizeof(float);
  int cap = (int)((48ull << 20) / (per_field ? per_field : 1));
  if (cap < 1) cap = 1;
  if (cap > work_fields) cap = work_fields;
  if (p->precision != DINO_PREC_FP32 && cap >= 64) {
    cap = cap / 64 * 64;
    const int chunks = (nf + cap - 1) / cap;
    const int even = (nf + chunks - 1) / chunks;
    return std::min(cap, (even + 63) / 64 * 64);
  }
  const int chunks = (nf + cap - 1) / cap;
  return (nf + chunks - 1) / chunks;
}

// Chunks alternate between the caller's stream and the plan's side stream
// when two of them fit in the workspace: each stream has its own half, both
// chunks' intermediates stay in L2, and one chunk's kernels fill the SMs the
// other leaves idle in its waves' tails.  The side stream forks from and joins back into the
// caller's stream with events, so the pattern also records into CUDA graphs.
struct ChunkRun {
  dino_plan* p;
  cudaStream_t st;
  float* work;
  size_t work_stride;  // floats per half
  bool dual = false;

  ChunkRun(dino_plan* p_, cudaStream_t st_, float* work_, int chunk, int nf,
           int work_fields)
      : p(p_), st(st_), work(work_), work_stride((size_t)chunk * p_->M * p_->J) {
    dual = p->side && nf > chunk && 2 * chunk <= work_fields;
  }
  int begin() {
    if (!dual) return DINO_OK;
    DINO_CHECK_CUDA(cudaEventRecord(p->ev_fork, st));
    DINO_CHECK_CUDA(cudaStreamWaitEvent(p->side, p->ev_fork, 0));
    return DINO_OK;
  }
  int slot(int c) const { return dual ? (c & 1) : -1; }
  cudaStream_t stream(int c) const { return slot(c) == 1 ? p->side : st; }
  float* buf(int c) const { return work + (slot(c) == 1 ? work_stride : 0); }
  int end() {
    if (!dual) return DINO_OK;
    DINO_CHECK_CUDA(cudaEventRecord(p->ev_join, p->side));
    DINO_CHECK_CUDA(cudaStreamWaitEvent(st, p->ev_join, 0));
    return DINO_OK;
  }
};

int sht_inverse_segs(dino_plan* p, const Segs& in, float* out, int nf,
                     float* work, int work_fields, cudaStream_t st) {
  const size_t ms = (size_t)p->M * p->L, ns = (size_t)p->I * p->J;
  const int chunk = l2_chunk(p, nf, work_fields);
  ChunkRun run(p, st, work, chunk, nf, work_fields);
  DINO_TRY(run.begin());
  for (int c = 0, f0 = 0; f0 < nf; ++c, f0 += chunk) {
    int n = nf - f0 < chunk ? nf - f0 : chunk;
    Segs sub = seg_offset(in, f0, n, ms);
    DINO_TRY(legendre_inverse(p, sub, run.buf(c), n, run.stream(c)));
    DINO_TRY(fourier_inverse(p, run.buf(c), out + f0 * ns, n, false, run.stream(c)));
  }
  return run.end();
}

int sht_forward_to(dino_plan* p, const float* nodal, float* out, int nf,
                   float* work, int work_fields, cudaStream_t st) {
  const size_t ms = (size_t)p->M * p->L, ns = (size_t)p->I * p->J;
  const int chunk = l2_chunk(p, nf, work_fields);
  ChunkRun run(p, st, work, chunk, nf, work_fields);
  DINO_TRY(run.begin());
  for (int c = 0, f0 = 0; f0 < nf; ++c, f0 += chunk) {
    int n = nf - f0 < chunk ? nf - f0 : chunk;
    DINO_TRY(fourier_forward(p, nodal + f0 * ns, run.buf(c), n, true, run.stream(c)));
    DINO_TRY(legendre_forward(p, run.buf(c), out + f0 * ms, n, run.stream(c)));
  }
  return run.end();
}

// Adjoint of the inverse transform: unweighted forward Fourier, then the
// forward contraction.  Adjoint of the forward transform: the inverse
// contraction, then the inverse Fourier synthesis scaled by w[j].  Chunked
// like the transforms themselves (work holds work_fields x M x J floats).
int sht_inverse_adjoint_to(dino_plan* p, const float* nodal_ct, float* modal_ct,
                           int nf, float* work, int work_fields, cudaStream_t st) {
  const size_t ms = (size_t)p->M * p->L, ns = (size_t)p->I * p->J;
  const int chunk = l2_chunk(p, nf, work_fields);
  ChunkRun run(p, st, work, chunk, nf, work_fields);
  DINO_TRY(run.begin());
  for (int c = 0, f0 = 0; f0 < nf; ++c, f0 += chunk) {
    int n = nf - f0 < chunk ? nf - f0 : chunk;
    DINO_TRY(fourier_forward(p, nodal_ct + f0 * ns, run.buf(c), n, false, run.stream(c)));
    DINO_TRY(legendre_forward(p, run.buf(c), modal_ct + f0 * ms, n, run.stream(c)));
  }
  return run.end();
}

int sht_forward_adjoint_to(dino_plan* p, const float* modal_ct, float* nodal_ct,
                           int nf, float* work, int work_fields, cudaStream_t st) {
  const size_t ms = (size_t)p->M * p->L, ns = (size_t)p->I * p->J;
  const int chunk = l2_chunk(p, nf, work_fields);
  ChunkRun run(p, st, work, chunk, nf, work_fields);
  DINO_TRY(run.begin());
  for (int c = 0, f0 = 0; f0 < nf; ++c, f0 += chunk) {
    int n = nf - f0 < chunk ? nf - f0 : chunk;
    DINO_TRY(legendre_inverse(p, one_seg(modal_ct + f0 * ms, n), run.buf(c), n,
                              run.stream(c)));
    DINO_TRY(fourier_inverse(p, run.buf(c), nodal_ct + f0 * ns, n, true, run.stream(c)));
  }
  return run.end();
}

static int sht_inverse_adjoint(dino_plan* p, const float* nodal_ct,
                               float* modal_ct, int nf, cudaStream_t st) {
  return sht_inverse_adjoint_to(p, nodal_ct, modal_ct, nf, p->d_work,
                                p->max_fields, st);
}

static int sht_forward_adjoint(dino_plan* p, const float* modal_ct,
                               float* nodal_ct, int nf, cudaStream_t st) {
  return sht_forward_adjoint_to(p, modal_ct, nodal_ct, nf, p->d_work,
                                p->max_fields, st);
}

// ---------------------------------------------------------------------------
// FastSphericalHarmonics modal layout (spherical_harmonic.py:411-621)
// ---------------------------------------------------------------------------

// Rows of the Fast layout are m = 0, 0 (imaginary, always zero), 1, -1, 2,
// -2, ... (:486-497): the Real layout [M = 2 lw - 1][L] with a zero row
// inserted at index 1.  to_fast: [M][L] -> [M + 1][L]; else the inverse
// (which drops row 1).
__global__ void modal_relayout_kernel(const float* __restrict__ in,
                                      float* __restrict__ out, int M, int L,
                                      int to_fast) {
  const int rows_in = to_fast ? M : M + 1, rows_out = to_fast ? M + 1 : M;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)rows_out * L) return;
  const int r = idx / L, l = idx % L;
  const float* src = in + (size_t)blockIdx.y * rows_in * L;
  float v;
  if (to_fast)
    v = (r == 0) ? src[l] : (r == 1 ? 0.f : src[(size_t)(r - 1) * L + l]);
  else
    v = src[(size_t)(r == 0 ? 0 : r + 1) * L + l];
  out[(size_t)blockIdx.y * rows_out * L + idx] = v;
}

int modal_relayout(dino_plan* p, bool to_fast, const float* in, float* out, int nf,
                   cudaStream_t st) {
  const int rows_out = to_fast ? p->M + 1 : p->M;
  dim3 grid(ceil_div(rows_out * p->L, 256), nf);
  modal_relayout_kernel<<<grid, 256, 0, st>>>(in, out, p->M, p->L, to_fast ? 1 : 0);
  return check_launch("modal_relayout");
}

// ---------------------------------------------------------------------------
// Spectral operators (spherical_harmonic.py:1033-1102)
// ---------------------------------------------------------------------------

// Spectral operators; `transpose` applies the transposed (adjoint) map.
// cos_lat_d_dlat: out[l] = ta[l+1] x[l+1] + tb[l-1] x[l-1]
//   transpose:    out[l] = ta[l] x[l-1] + tb[l] x[l+1]
// d_dlon is antisymmetric; the Laplacians and the clip are diagonal.
__global__ void modal_op_kernel(int op, int transpose,
                                const float* __restrict__ in,
                                float* __restrict__ out, int nf, int M, int L,
                                int lw, const float* __restrict__ deriv,
                                const float* __restrict__ lap,
                                const float* __restrict__ invlap, int clip_n) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t total = (size_t)nf * M * L;
  if (idx >= total) return;
  int l = idx % L;
  int row = (idx / L) % M;
  size_t base = idx - l - (size_t)row * L;  // start of this field
  int m = (row + 1) / 2;
  const float* x = in + base;
  float v = 0.f;
  switch (op) {
    case DINO_OP_D_DLON: {
      float s = transpose ? -1.f : 1.f;
      if (row == 0) v = 0.f;
      else if (row & 1) v = s * m * x[(size_t)(row + 1) * L + l];
      else v = -s * m * x[(size_t)(row - 1) * L + l];
      break;
    }
    case DINO_OP_COS_LAT_D_DLAT:
    case DINO_OP_SEC_LAT_D_DLAT_COS2: {
      const float* ta = deriv + (op == DINO_OP_COS_LAT_D_DLAT ? 0 : 2) * (size_t)lw * L;
      const float* tb = ta + (size_t)lw * L;
      const float* xr = x + (size_t)row * L;
      const float* tam = ta + (size_t)m * L;
      const float* tbm = tb + (size_t)m * L;
      if (!transpose) {
        if (l + 1 < L) v += tam[l + 1] * xr[l + 1];
        if (l >= 1) v += tbm[l - 1] * xr[l - 1];
      } else {
        if (l >= 1) v += tam[l] * xr[l - 1];
        if (l + 1 < L) v += tbm[l] * xr[l + 1];
      }
      break;
    }
    case DINO_OP_LAPLACIAN:
      v = x[(size_t)row * L + l] * lap[l];
      break;
    case DINO_OP_INVERSE_LAPLACIAN:
      v = x[(size_t)row * L + l] * invlap[l];
      break;
    case DINO_OP_CLIP:
      v = (l < L - clip_n) ? x[(size_t)row * L + l] : 0.f;
      break;
  }
  out[idx] = v;
}

int modal_op(dino_plan* p, int op, const float* in, float* out, int nf, int arg,
             cudaStream_t st) {
  const int transpose = (op & 8) ? 1 : 0;
  op &= 7;
  DINO_REQUIRE(op >= DINO_OP_D_DLON && op <= DINO_OP_CLIP, DINO_ERR_ARG,
               "unknown modal operator");
  DINO_REQUIRE(op != DINO_OP_CLIP || arg > 0, DINO_ERR_ARG,
               "`n` must be >= 0");
  DINO_REQUIRE(in != out, DINO_ERR_ARG, "modal_op: in and out must differ");
  size_t total = (size_t)nf * p->M * p->L;
  if (total == 0) return DINO_OK;
  modal_op_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(
      op, transpose, in, out, nf, p->M, p->L, p->lw, p->d_deriv, p->d_lap,
      p->d_invlap, arg);
  return check_launch("modal_op");
}

}  // namespace dino

using namespace dino;

extern "C" {

int dino_sht_inverse(dino_plan* p, const float* modal, float* nodal, int32_t nf,
                     void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "dino_sht_inverse: null plan");
  DINO_REQUIRE(nf >= 0, DINO_ERR_SHAPE, "nfields must be >= 0");
  if (nf == 0) return DINO_OK;  // buffers may be null for an empty batch
  DINO_REQUIRE(modal && nodal, DINO_ERR_ARG, "dino_sht_inverse: null argument");
  return sht_inverse_segs(p, one_seg(modal, nf), nodal, nf, p->d_work,
                          p->max_fields, (cudaStream_t)stream);
}

int dino_sht_forward(dino_plan* p, const float* nodal, float* modal, int32_t nf,
                     void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "dino_sht_forward: null plan");
  DINO_REQUIRE(nf >= 0, DINO_ERR_SHAPE, "nfields must be >= 0");
  if (nf == 0) return DINO_OK;
  DINO_REQUIRE(modal && nodal, DINO_ERR_ARG, "dino_sht_forward: null argument");
  return sht_forward_to(p, nodal, modal, nf, p->d_work, p->max_fields,
                        (cudaStream_t)stream);
}

int dino_sht_inverse_adjoint(dino_plan* p, const float* nodal_ct,
                             float* modal_ct, int32_t nf, void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "null plan");
  DINO_REQUIRE(nf >= 0, DINO_ERR_SHAPE, "nfields must be >= 0");
  if (nf == 0) return DINO_OK;
  DINO_REQUIRE(nodal_ct && modal_ct, DINO_ERR_ARG, "null argument");
  return sht_inverse_adjoint(p, nodal_ct, modal_ct, nf, (cudaStream_t)stream);
}

int dino_sht_forward_adjoint(dino_plan* p, const float* modal_ct,
                             float* nodal_ct, int32_t nf, void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "null plan");
  DINO_REQUIRE(nf >= 0, DINO_ERR_SHAPE, "nfields must be >= 0");
  if (nf == 0) return DINO_OK;
  DINO_REQUIRE(nodal_ct && modal_ct, DINO_ERR_ARG, "null argument");
  return sht_forward_adjoint(p, modal_ct, nodal_ct, nf, (cudaStream_t)stream);
}

int dino_sht_phase(dino_plan* p, int32_t phase, const float* in, float* out,
                   int32_t nf, void* stream) {
  DINO_REQUIRE(p && in && out, DINO_ERR_ARG, "dino_sht_phase: null argument");
  DINO_REQUIRE(nf >= 0 && nf <= p->max_fields, DINO_ERR_SHAPE,
               "nfields must be in [0, max_fields]");
  if (nf == 0) return DINO_OK;
  cudaStream_t st = (cudaStream_t)stream;
  switch (phase) {
    case DINO_PHASE_LEGENDRE_INVERSE:
      return legendre_inverse(p, one_seg(in, nf), out, nf, st);
    case DINO_PHASE_FOURIER_INVERSE:
      return fourier_inverse(p, in, out, nf, false, st);
    case DINO_PHASE_FOURIER_FORWARD:
      return fourier_forward(p, in, out, nf, true, st);
    case DINO_PHASE_LEGENDRE_FORWARD:
      return legendre_forward(p, in, out, nf, st);
  }
  set_error("unknown transform phase");
  return DINO_ERR_ARG;
}

int dino_modal_op(dino_plan* p, int32_t op, const float* in, float* out,
                  int32_t nf, int32_t arg, void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "dino_modal_op: null plan");
  DINO_REQUIRE(nf >= 0, DINO_ERR_SHAPE, "nfields must be >= 0");
  if (nf == 0) return DINO_OK;
  DINO_REQUIRE(in && out, DINO_ERR_ARG, "dino_modal_op: null argument");
  return modal_op(p, op, in, out, nf, arg, (cudaStream_t)stream);
}

int dino_modal_relayout(dino_plan* p, int32_t to_fast, const float* in, float* out,
                        int32_t nfields, void* stream) {
  DINO_REQUIRE(p, DINO_ERR_ARG, "dino_modal_relayout: null plan");
  DINO_REQUIRE(nfields >= 0 && nfields <= 65535, DINO_ERR_SHAPE, "nfields out of range");
  if (nfields == 0) return DINO_OK;
  DINO_REQUIRE(in && out, DINO_ERR_ARG, "dino_modal_relayout: null argument");
  DINO_REQUIRE(in != out, DINO_ERR_ARG, "dino_modal_relayout: in and out must differ");
  return modal_relayout(p, to_fast != 0, in, out, nfields, (cudaStream_t)stream);
}

}  // extern "C"
