// On-the-fly Nyström pair product y = A x, A_ij = K(x_i, y_j) w_j
// (src/nystrom.jl:93-96 entries; src/nystrom.jl:117-124 is the CPU loop it
// replaces), for the Laplace (2D/3D) and Helmholtz (3D) single-layer,
// double-layer, adjoint-double-layer and hypersingular kernels
// (src/kernels.jl:137-204, 347-413).
//
// Design (B200, sm_100a):
//  * A pack kernel folds the density into per-source records
//    (coordinates + w*sigma, or the dipole w*sigma*n for DL/HS), padded to
//    whole tiles with zero charges.
//  * The pair kernel gives each thread TPT targets held in registers.  Source
//    tiles are streamed into shared memory by the TMA bulk-copy engine
//    (cp.async.bulk + mbarrier, two stages, one elected thread issues) and
//    read back as broadcasts.  Each CTA covers one target block and one chunk
//    of the source tiles (grid.y = split), so every SM stays busy even when
//    the target count is small; partial sums go to scratch and are reduced in
//    a fixed order by the epilogue (deterministic, no atomics).
//  * FP64 form: FP64 pairs and sums.  FP32C form: FP32 pairs, summed in FP32
//    over groups of 32 sources, groups folded into a (sum, compensation)
//    pair with Knuth's TwoSum (error-free), so the long sum over N sources
//    carries no O(N eps) growth.
//  * The epilogue applies the kernel constant, alpha/beta, and the CSR
//    correction row in the same pass (the fused near-field correction).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "common.h"
#include "device_common.cuh"

namespace inti {

constexpr int kBlock = 128;  // threads per CTA
constexpr int kTPT = 4;      // targets per thread
constexpr int kTile64 = 128; // sources per shared-memory stage (FP64)
constexpr int kFineTile = 32;  // sources per stage where whole tiles leave SMs idle (FP64)
constexpr int kTile32 = 256; // sources per shared-memory stage (FP32C)
constexpr int kGroup = 32;   // FP32C: sources summed before a compensated fold

// ---------------------------------------------------------------------------
// Source record layouts (elements of R per source):
//   Laplace  SL/ADL : x y [z] q            (q = w*sigma)
//   Laplace  DL/HS  : x y [z] p_x p_y [p_z] (p = w*sigma*n_y)
//   Helmholtz SL/ADL: x y z qr qi
//   Helmholtz DL/HS : x y z pr_x pr_y pr_z pi_x pi_y pi_z
// each padded so that a record is a multiple of 16 bytes.
// ---------------------------------------------------------------------------
//   combined field (CF): x y z | dipole c1*w*sigma*n_y | charge c2*w*sigma
template <int PDE, int KIND, int DIM, class R>
struct Rec {
  static constexpr bool dipole = (KIND == DL || KIND == HS || KIND == CF);
  static constexpr bool charge2 = (KIND == CF);
  static constexpr bool cplx = (PDE == HELMHOLTZ);
  static constexpr int used = DIM + (cplx ? 2 : 1) * ((dipole ? DIM : 1) + (charge2 ? 1 : 0));
  static constexpr int align = 16 / sizeof(R);
  static constexpr int n = (used + align - 1) / align * align;
  static constexpr bool tnormal = (KIND == ADL || KIND == HS);
};

// Record of source j (zero past n: a zero charge at the origin, which adds
// nothing to any target).
template <int PDE, int KIND, int DIM, class R>
__device__ __forceinline__ void build_record(int64_t j, int64_t n, const double* __restrict__ xs,
                                             const double* __restrict__ ns, const double* __restrict__ w,
                                             const double* __restrict__ sigma, double2 c1, double2 c2,
                                             R (&rec)[Rec<PDE, KIND, DIM, R>::n]) {
  using RC = Rec<PDE, KIND, DIM, R>;
#pragma unroll
  for (int c = 0; c < RC::n; ++c) rec[c] = R(0);
  if (j >= n) return;
#pragma unroll
  for (int c = 0; c < DIM; ++c) rec[c] = R(xs[DIM * j + c]);
  const double wj = w[j];
  double qr, qi = 0.0;
  if (RC::cplx) {
    qr = wj * sigma[2 * j];
    qi = wj * sigma[2 * j + 1];
  } else {
    qr = wj * sigma[j];
  }
  if (RC::charge2) {
    // monopole charge c2*q after the dipole block
    const double mr = c2.x * qr - c2.y * qi, mi = c2.x * qi + c2.y * qr;
    rec[DIM + (RC::cplx ? 2 : 1) * DIM] = R(mr);
    if (RC::cplx) rec[DIM + 2 * DIM + 1] = R(mi);
    const double dr = c1.x * qr - c1.y * qi, di = c1.x * qi + c1.y * qr;
    qr = dr;
    qi = di;
  }
  if (RC::dipole) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      rec[DIM + c] = R(qr * ns[DIM * j + c]);
      if (RC::cplx) rec[2 * DIM + c] = R(qi * ns[DIM * j + c]);
    }
  } else {
    rec[DIM] = R(qr);
    if (RC::cplx) rec[DIM + 1] = R(qi);
  }
}

template <int PDE, int KIND, int DIM, class R>
__global__ void pack_sources(int64_t n, int64_t npad, const double* __restrict__ xs,
                             const double* __restrict__ ns, const double* __restrict__ w,
                             const double* __restrict__ sigma, double2 c1, double2 c2,
                             R* __restrict__ out) {
  using RC = Rec<PDE, KIND, DIM, R>;
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (j >= npad) return;
  R rec[RC::n];
  build_record<PDE, KIND, DIM, R>(j, n, xs, ns, w, sigma, c1, c2, rec);
  R* o = out + j * RC::n;
#pragma unroll
  for (int c = 0; c < RC::n; ++c) o[c] = rec[c];
}

// ---------------------------------------------------------------------------
// Per-pair accumulation.  Kernel constants (1/(4pi), signs) are applied once
// in the epilogue; the self pair (|r|^2 <= tol^2) contributes exactly zero.
// ---------------------------------------------------------------------------
template <class R>
struct MathOps;
template <>
struct MathOps<double> {
  using R2 = double2;
  static __device__ __forceinline__ double rsq(double v) { return rsqrt_fast(v); }
  static __device__ __forceinline__ double rsq3(double v) { return rsqrt_cube_fast(v); }
  static __device__ __forceinline__ double rcp(double v) { return rcp_fast(v); }
  static __device__ __forceinline__ double lg(double v) { return log(v); }
  static __device__ __forceinline__ bool keep(double d2) { return pair_keep(d2); }
};
template <>
struct MathOps<float> {
  using R2 = float2;
  static __device__ __forceinline__ float rsq(float v) { return rsqrt_fast(v); }
  static __device__ __forceinline__ float rsq3(float v) { return rsqrt_cube_fast(v); }
  static __device__ __forceinline__ float rcp(float v) { return 1.0f / v; }
  static __device__ __forceinline__ float lg(float v) { return __logf(v); }
  static __device__ __forceinline__ bool keep(float d2) { return d2 > 1.0e-28f; }
};

template <class R, int DIM, bool TN>
struct Target {
  R x[DIM];
  R n[TN ? DIM : 1];
};

// Helmholtz phase: e^{ikd} = expi(d * kT) with kT = k*kExpiTable/(2 pi)
// (table + Taylor, see expi_table_eval).
struct HelmConst {
  double kT, delta;
};

template <int PDE, int KIND, int DIM, class R>
__device__ __forceinline__ void pair_step(const Target<R, DIM, Rec<PDE, KIND, DIM, R>::tnormal>& t,
                                          const R* __restrict__ s, R kT, R delta, R k,
                                          const typename MathOps<R>::R2* __restrict__ tab, R& ar, R& ai) {
  using M = MathOps<R>;
  R r[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) r[c] = t.x[c] - s[c];
  R d2 = r[0] * r[0];
#pragma unroll
  for (int c = 1; c < DIM; ++c) d2 = fma(r[c], r[c], d2);
  const bool keep = M::keep(d2);
  if (PDE == LAPLACE) {
    if (KIND == SL) {
      if (DIM == 2) {
        // -log(d)/(2pi) = log(d^2) * (-1/(4pi)); constant in the epilogue
        const R l = M::lg(d2);
        ar += keep ? l * s[2] : R(0);
      } else {
        const R ri = keep ? M::rsq(d2) : R(0);
        ar = fma(ri, s[3], ar);
      }
    } else if (KIND == DL || KIND == CF) {
      R rp = r[0] * s[DIM];
#pragma unroll
      for (int c = 1; c < DIM; ++c) rp = fma(r[c], s[DIM + c], rp);
      if (DIM == 2) {
        const R ri = keep ? M::rcp(d2) : R(0);
        ar = fma(rp, ri, ar);
      } else if (KIND == CF) {
        const R ri = keep ? M::rsq(d2) : R(0);
        ar = fma(ri, s[2 * DIM], ar);
        ar = fma(rp, ri * ri * ri, ar);
      } else {
        ar = fma(rp, keep ? M::rsq3(d2) : R(0), ar);
      }
    } else if (KIND == ADL) {
      R rn = r[0] * t.n[0];
#pragma unroll
      for (int c = 1; c < DIM; ++c) rn = fma(r[c], t.n[c], rn);
      const R q = s[DIM];
      if (DIM == 2) {
        const R ri = keep ? M::rcp(d2) : R(0);
        ar = fma(rn * q, ri, ar);
      } else {
        ar = fma(rn * q, keep ? M::rsq3(d2) : R(0), ar);
      }
    } else {  // HS: (nx.p - DIM (r.nx)(r.p)/d^2) / d^DIM
      R rn = r[0] * t.n[0], rp = r[0] * s[DIM], np = t.n[0] * s[DIM];
#pragma unroll
      for (int c = 1; c < DIM; ++c) {
        rn = fma(r[c], t.n[c], rn);
        rp = fma(r[c], s[DIM + c], rp);
        np = fma(t.n[c], s[DIM + c], np);
      }
      if (DIM == 2) {
        const R id2 = keep ? M::rcp(d2) : R(0);
        ar = fma(id2, fma(R(-2) * rn * rp, id2, np), ar);
      } else {
        const R ri = keep ? M::rsq(d2) : R(0);
        const R id2 = ri * ri;
        ar = fma(id2 * ri, fma(R(-3) * rn * rp, id2, np), ar);
      }
    }
  } else {  // Helmholtz 3D
    const R ri = keep ? M::rsq(d2) : R(0);
    const R d = d2 * ri;  // 0 for the self pair
    R sn, cs;
    expi_table_eval(d, kT, tab, delta, cs, sn);
    if (KIND == SL || KIND == ADL) {
      R g_r, g_i;  // G (without 1/4pi) or the ADL factor
      if (KIND == SL) {
        g_r = ri * cs;
        g_i = ri * sn;
      } else {
        // e^{ikd}(1/d - ik) (r.nx) / d^2
        const R er = fma(cs, ri, k * sn), ei = fma(sn, ri, -k * cs);
        R rn = r[0] * t.n[0];
        rn = fma(r[1], t.n[1], rn);
        rn = fma(r[2], t.n[2], rn);
        const R f = rn * ri * ri;
        g_r = er * f;
        g_i = ei * f;
      }
      const R qr = s[3], qi = s[4];
      ar = fma(g_r, qr, fma(-g_i, qi, ar));
      ai = fma(g_r, qi, fma(g_i, qr, ai));
    } else if (KIND == DL || KIND == CF) {
      const R er = fma(cs, ri, k * sn), ei = fma(sn, ri, -k * cs);
      const R id2 = ri * ri;
      R A = r[0] * s[3], B = r[0] * s[6];
      A = fma(r[1], s[4], A);
      A = fma(r[2], s[5], A);
      B = fma(r[1], s[7], B);
      B = fma(r[2], s[8], B);
      const R gr = er * id2, gi = ei * id2;
      ar = fma(gr, A, fma(-gi, B, ar));
      ai = fma(gr, B, fma(gi, A, ai));
      if (KIND == CF) {  // + e^{ikd}/d * (c2 w sigma)
        const R hr = cs * ri, hi = sn * ri;
        const R qr = s[9], qi = s[10];
        ar = fma(hr, qr, fma(-hi, qi, ar));
        ai = fma(hr, qi, fma(hi, qr, ai));
      }
    } else {  // HS
      const R id2 = ri * ri;
      R rn = r[0] * t.n[0];
      rn = fma(r[1], t.n[1], rn);
      rn = fma(r[2], t.n[2], rn);
      R A = r[0] * s[3], B = r[0] * s[6], NA = t.n[0] * s[3], NB = t.n[0] * s[6];
#pragma unroll
      for (int c = 1; c < 3; ++c) {
        A = fma(r[c], s[3 + c], A);
        B = fma(r[c], s[6 + c], B);
        NA = fma(t.n[c], s[3 + c], NA);
        NB = fma(t.n[c], s[6 + c], NB);
      }
      // value = a (r.nx)(r.p) + b (nx.p) with b = e^{ikd}(1/d - ik)/d^2,
      // a = e^{ikd}(k^2 d^2 - 3 + 3ikd)/d^5 and the complex dipole sums
      // r.p = A + iB, nx.p = NA + iNB; formed as e^{ikd} W with
      // W = (k^2 d^2 - 3 + 3ikd) U + (1/d - ik) P, U = (r.nx)(A + iB)/d^5,
      // P = (NA + iNB)/d^2
      const R kd = k * d;
      const R fr = fma(kd, kd, R(-3)), fi = R(3) * kd;
      const R u = rn * (id2 * id2 * ri);
      const R ur = u * A, ui = u * B, pr = NA * id2, pi = NB * id2;
      const R wr = fma(fr, ur, fma(-fi, ui, fma(ri, pr, k * pi)));
      const R wi = fma(fr, ui, fma(fi, ur, fma(ri, pi, -k * pr)));
      ar = fma(cs, wr, fma(-sn, wi, ar));
      ai = fma(cs, wi, fma(sn, wr, ai));
    }
  }
}

// Accumulator: FP64 plain; FP32 with a per-group sum and a TwoSum-folded
// (hi, lo) pair.
template <class R, bool CPLX>
struct Acc;
template <bool CPLX>
struct Acc<double, CPLX> {
  double r = 0, i = 0;
  __device__ __forceinline__ double& gr() { return r; }
  __device__ __forceinline__ double& gi() { return i; }
  __device__ __forceinline__ void fold() {}
};
__device__ __forceinline__ void two_sum_fold(float& hi, float& lo, float& g) {
  const float t = hi + g;
  const float bp = t - hi;
  const float e = (hi - (t - bp)) + (g - bp);
  hi = t;
  lo += e;
  g = 0.f;
}
template <bool CPLX>
struct Acc<float, CPLX> {
  float gr_ = 0, gi_ = 0, hr = 0, lr = 0, hi = 0, li = 0;
  __device__ __forceinline__ float& gr() { return gr_; }
  __device__ __forceinline__ float& gi() { return gi_; }
  __device__ __forceinline__ void fold() {
    two_sum_fold(hr, lr, gr_);
    if (CPLX) two_sum_fold(hi, li, gi_);
  }
};

// Partial accumulator storage per (split, target).
template <class R, bool CPLX>
struct PartialT;
template <>
struct PartialT<double, false> { using T = double; };
template <>
struct PartialT<double, true> { using T = double2; };
template <>
struct PartialT<float, false> { using T = float2; };
template <>
struct PartialT<float, true> { using T = float4; };

__device__ __forceinline__ void store_partial(double* p, const Acc<double, false>& a) { *p = a.r; }
__device__ __forceinline__ void store_partial(double2* p, const Acc<double, true>& a) {
  *p = make_double2(a.r, a.i);
}
__device__ __forceinline__ void store_partial(float2* p, const Acc<float, false>& a) {
  *p = make_float2(a.hr, a.lr);
}
__device__ __forceinline__ void store_partial(float4* p, const Acc<float, true>& a) {
  *p = make_float4(a.hr, a.lr, a.hi, a.li);
}
__device__ __forceinline__ void add_partial(Acc<double, false>& a, double p) { a.r += p; }
__device__ __forceinline__ void add_partial(Acc<double, true>& a, double2 p) {
  a.r += p.x;
  a.i += p.y;
}

// Slices of a CTA of pair_forward.  FP64: the four warps have the same targets
// and a quarter of a tile's sources each, so that few targets still make many
// CTAs and their chunks' partial sums stay four times fewer.  What bounds the
// kernel is the FP64 pipe once an SM has some 12 CTAs; below that, idle SMs
// and latency.  With a target block per warp and thread-per-row epilogues,
// products back to back, Laplace DL: 51,894 sources x 4,096 / 1,000 / 100
// targets 280 / 113 / 105 us, 3,456 x 1,000 51.2; now 248 / 70 / 20 and 12.1.
// FP32C keeps one slice: its groups of sums are folded in the order of the
// tile.
template <class R>
constexpr int fwd_slices() {
  return std::is_same<R, float>::value ? 1 : kBlock / 32;
}
// Targets per CTA of pair_forward.
static int64_t fwd_rows(int precision, int tpt) {
  return (int64_t)tpt * kBlock / (precision == INTI_FP32C ? fwd_slices<float>() : fwd_slices<double>());
}

struct FwdArgs {
  int64_t m;
  int64_t n_tiles;
  int tiles_per_split;
  const double* tcoords;
  const double* tnormals;
  const void* packed;
  void* partial;
  double k;
  double kT, delta;   // Helmholtz phase scaling (see HelmConst)
  const void* expi;   // kExpiTable (cos, sin) entries in R precision
  int* err;
};

// CTAs per SM that the FP64 pair kernels ask the compiler for: one lets it
// take the registers that keep more pairs in flight, zero leaves its own
// choice (more CTAs).  Which is faster depends on the arithmetic of a pair,
// so it is measured per kernel.  Symmetric form, 19,200 nodes, zero -> as
// below, us: Laplace 3D SL 219 -> 200, HS 406 -> 391; 2D ADL 245 -> 234,
// HS 301 -> 278; Helmholtz SL 522 -> 488, ADL 711 -> 698, HS 806 -> 786, CF
// 857 -> 854 (two targets per thread 899 -> 854).  Slower with one, so left at
// zero: Laplace 3D DL 318 (347), ADL 342 (369), CF 344 (351), 2D SL 662
// (683), Helmholtz DL 725 (741).  One-sided, 3,888 targets x 12,288 sources:
// Laplace 3D SL 54 -> 49, HS 100 -> 96, 2D DL 47 -> 43, ADL 49 -> 47, HS 71 ->
// 67, Helmholtz SL 124 -> 116, DL 155 -> 153, ADL 153 -> 144.
template <int PDE, int KIND, int DIM, class R>
constexpr int fwd_min_ctas() {
  if (std::is_same<R, float>::value || KIND == CF) return 0;
  return PDE == HELMHOLTZ || (DIM == 3 ? KIND == SL || KIND == HS : KIND != SL) ? 1 : 0;
}
template <int PDE, int KIND, int DIM, class R>
constexpr int symm_min_ctas() {
  if (std::is_same<R, float>::value) return 0;
  if (PDE == HELMHOLTZ) return KIND == DL ? 0 : KIND == CF ? 3 : 1;
  return fwd_min_ctas<PDE, KIND, DIM, R>();
}

template <int PDE, int KIND, int DIM, class R, int TILE, int TPT = kTPT>
__global__ void __launch_bounds__(kBlock, (fwd_min_ctas<PDE, KIND, DIM, R>())) pair_forward(FwdArgs a) {
  using RC = Rec<PDE, KIND, DIM, R>;
  constexpr bool CPLX = RC::cplx;
  using P = typename PartialT<R, CPLX>::T;
  using R2 = typename MathOps<R>::R2;
  constexpr uint32_t kStageBytes = TILE * RC::n * sizeof(R);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* stage0 = reinterpret_cast<R*>(smem_raw);
  R* stage1 = reinterpret_cast<R*>(smem_raw + kStageBytes);
  R2* tab = reinterpret_cast<R2*>(smem_raw + 2 * kStageBytes);  // Helmholtz only
  __shared__ __align__(8) uint64_t full[2];

  const int tid = threadIdx.x;
  constexpr int NSL = fwd_slices<R>(), kRows = kBlock / NSL;  // a slice's threads: one target each, TPT times
  const int row = tid % kRows, slice = tid / kRows;
  const int64_t base = (int64_t)blockIdx.x * (kRows * TPT);
  const int split = blockIdx.y;
  const int64_t t0 = (int64_t)split * a.tiles_per_split;
  const int64_t t1 = min(a.n_tiles, t0 + a.tiles_per_split);
  const R* src = static_cast<const R*>(a.packed);

  pdl_trigger();
  Target<R, DIM, RC::tnormal> tg[TPT];
  Acc<R, CPLX> acc[TPT];
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
    const int64_t i = min(base + u * kRows + row, a.m - 1);
#pragma unroll
    for (int c = 0; c < DIM; ++c) tg[u].x[c] = R(a.tcoords[DIM * i + c]);
    if (RC::tnormal) {
#pragma unroll
      for (int c = 0; c < DIM; ++c) tg[u].n[c] = R(a.tnormals[DIM * i + c]);
    }
  }
  const R k = R(a.k);
  const R kT = R(a.kT);
  const R delta = R(a.delta);
  if (RC::cplx) {
    const R2* g = static_cast<const R2*>(a.expi);
    for (int q = tid; q < kExpiTable; q += kBlock) tab[q] = g[q];
  }

  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();  // the packed records; the partials of the product before are consumed
  int64_t issued = t0;  // next tile to issue (meaningful in thread 0)
  if (tid == 0) {
    for (int s = 0; s < 2 && issued < t1; ++s, ++issued) {
      mbar_arrive_expect_tx(&full[s], kStageBytes);
      bulk_copy_g2s(s ? stage1 : stage0, src + issued * TILE * RC::n, kStageBytes, &full[s]);
    }
  }

  for (int64_t t = t0; t < t1; ++t) {
    const int st = (int)((t - t0) & 1);
    const uint32_t parity = (uint32_t)(((t - t0) >> 1) & 1);
    const bool ok = mbar_wait_bounded(&full[st], parity);
    if (!__syncthreads_and(ok)) {
      // A bulk copy never completed: record it, drain what is still in
      // flight (bounded), and leave without touching the results.
      if (tid == 0) {
        atomicExch(a.err, kErrWaitTimeout);
        for (int64_t q = t + 1; q < issued; ++q)
          mbar_wait_bounded(&full[(q - t0) & 1], (uint32_t)(((q - t0) >> 1) & 1));
      }
      return;
    }
    const R* sp = st ? stage1 : stage0;
    constexpr int kShare = TILE / NSL, kRun = kShare < kGroup ? kShare : kGroup;
#pragma unroll 1
    for (int g = slice * kShare; g < (slice + 1) * kShare; g += kRun) {
#pragma unroll 2
      for (int s = 0; s < kRun; ++s) {
        const R* rec = sp + (g + s) * RC::n;
#pragma unroll
        for (int u = 0; u < TPT; ++u)
          pair_step<PDE, KIND, DIM, R>(tg[u], rec, kT, delta, k, tab, acc[u].gr(), acc[u].gi());
      }
#pragma unroll
      for (int u = 0; u < TPT; ++u) acc[u].fold();
    }
    __syncthreads();  // every thread is done reading this stage
    if (tid == 0 && issued < t1) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[st], kStageBytes);
      bulk_copy_g2s(st ? stage1 : stage0, src + issued * TILE * RC::n, kStageBytes, &full[st]);
      ++issued;
    }
  }
  P* out = static_cast<P*>(a.partial) + (int64_t)split * a.m;
  if constexpr (NSL > 1) {
    // the slices' sums, added in a fixed order (the stages are free: every
    // tile issued was waited for)
    static_assert((NSL - 1) * kRows * TPT * sizeof(P) <= 2 * kStageBytes, "the slices' sums fit the stages");
    P* red = reinterpret_cast<P*>(smem_raw);
#pragma unroll
    for (int u = 0; u < TPT; ++u)
      if (slice > 0) store_partial(red + ((slice - 1) * TPT + u) * kRows + row, acc[u]);
    __syncthreads();
    if (slice > 0) return;
#pragma unroll
    for (int u = 0; u < TPT; ++u)
      for (int q = 1; q < NSL; ++q) add_partial(acc[u], red[((q - 1) * TPT + u) * kRows + row]);
  }
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
    const int64_t i = base + u * kRows + row;
    if (i < a.m) store_partial(out + i, acc[u]);
  }
}

// ---------------------------------------------------------------------------
// Epilogue: y_i = alpha*(scale*sum_s partial[s][i] + sum_p C_ip x_p) + beta*y_i
// ---------------------------------------------------------------------------
__device__ __forceinline__ double2 load_partial(const double* p) { return make_double2(*p, 0.0); }
__device__ __forceinline__ double2 load_partial(const double2* p) { return *p; }
__device__ __forceinline__ double2 load_partial(const float2* p) {
  const float2 v = *p;
  return make_double2((double)v.x + (double)v.y, 0.0);
}
__device__ __forceinline__ double2 load_partial(const float4* p) {
  const float4 v = *p;
  return make_double2((double)v.x + (double)v.y, (double)v.z + (double)v.w);
}

struct EpiArgs {
  int64_t m;
  int split;
  const void* partial;
  double scale;
  const int64_t* rowptr;  // null when no correction
  const int32_t* col;
  const double* val;
  const double* x;
  double* y;
  double ar, ai, br, bi;
  bool beta_zero;
  const double* rowscale = nullptr;  // per-row factor of the pair sum (A^T: the source weights)
  const int* err = nullptr;          // when set and nonzero (a pair kernel timed out): y gets NaN
};

// y[i] before the product (read only when beta != 0).
template <bool CPLX>
__device__ __forceinline__ double2 epilogue_y_old(const EpiArgs& e, int64_t i) {
  return CPLX ? reinterpret_cast<const double2*>(e.y)[i] : make_double2(e.y[i], 0.0);
}

// y[i] = alpha * (sr, si) + beta * yo, yo the old y[i].
template <bool CPLX>
__device__ __forceinline__ void epilogue_store(const EpiArgs& e, int64_t i, double sr, double si, double2 yo) {
  if (CPLX) {
    double yr = e.ar * sr - e.ai * si, yi = e.ar * si + e.ai * sr;
    if (!e.beta_zero) {
      yr += e.br * yo.x - e.bi * yo.y;
      yi += e.br * yo.y + e.bi * yo.x;
    }
    reinterpret_cast<double2*>(e.y)[i] = make_double2(yr, yi);
  } else {
    double yr = e.ar * sr;
    if (!e.beta_zero) yr += e.br * yo.x;
    e.y[i] = yr;
  }
}

// y_i = alpha*(scale*pair sum + correction row) + beta*y_i for `nodes` rows per
// CTA, and for each as many threads as that leaves: thread
// sl of a row sums every slices-th chunk and correction entry, and the sums
// are added in a fixed order.
template <class P, bool CPLX>
__global__ void pair_epilogue_kernel(EpiArgs e, int nodes) {
  extern __shared__ double4 epi_part[];  // slices x nodes, for more than one slice
  const int tn = threadIdx.x % nodes, sl = threadIdx.x / nodes, slices = blockDim.x / nodes;
  const int64_t i = blockIdx.x * (int64_t)nodes + tn;
  pdl_trigger();
  pdl_wait();
  if (e.err && *e.err) {  // the partial sums are incomplete: make the failure visible in y
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    if (sl > 0 || i >= e.m) return;
    if (CPLX)
      reinterpret_cast<double2*>(e.y)[i] = make_double2(nan, nan);
    else
      e.y[i] = nan;
    return;
  }
  double4 c = make_double4(0.0, 0.0, 0.0, 0.0);  // pair sum, correction sum
  if (i < e.m) {
    const P* part = static_cast<const P*>(e.partial) + i;
#pragma unroll 4
    for (int s = sl; s < e.split; s += slices) {
      const double2 v = load_partial(part + (int64_t)s * e.m);
      c.x += v.x;
      c.y += v.y;
    }
    if (e.rowptr) {
      for (int64_t p = e.rowptr[i] + sl, p1 = e.rowptr[i + 1]; p < p1; p += slices) {
        const int32_t j = e.col[p];
        if (CPLX) {
          const double2 v = reinterpret_cast<const double2*>(e.val)[p];
          const double2 xv = reinterpret_cast<const double2*>(e.x)[j];
          c.z = fma(v.x, xv.x, fma(-v.y, xv.y, c.z));
          c.w = fma(v.x, xv.y, fma(v.y, xv.x, c.w));
        } else {
          c.z = fma(e.val[p], e.x[j], c.z);
        }
      }
    }
  }
  if (slices > 1) {
    epi_part[threadIdx.x] = c;
    __syncthreads();
    if (sl > 0) return;
    for (int q = 1; q < slices; ++q) {
      const double4 v = epi_part[q * nodes + tn];
      c.x += v.x;
      c.y += v.y;
      c.z += v.z;
      c.w += v.w;
    }
  }
  if (i >= e.m) return;
  const double sc = e.rowscale ? e.scale * e.rowscale[i] : e.scale;
  epilogue_store<CPLX>(e, i, fma(c.x, sc, c.z), fma(c.y, sc, c.w),
                       e.beta_zero ? make_double2(0.0, 0.0) : epilogue_y_old<CPLX>(e, i));
}

struct EpiShape {
  int nodes, slices;
  unsigned threads() const { return (unsigned)(nodes * slices); }
  unsigned blocks(int64_t m) const { return (unsigned)((m + nodes - 1) / nodes); }
  size_t smem() const { return slices > 1 ? sizeof(double4) * threads() : 0; }
};
// The rows of few chunks have enough threads with one each; with more, a
// row's chunks are one long chain of loads and are split over 8 or 32
// (1,000 rows: 203 chunks 31.8 us with a thread per row, 406 chunks 6.6 with 32).
static EpiShape epi_shape(int split) {
  if (split < 8) return {256, 1};
  return {32, split < 64 ? 8 : 32};
}

// ---------------------------------------------------------------------------
// Single-launch form for small FP64 operators (m*n up to kSmallPairs, e.g.
// the 1,000-node kite): one kernel per product, no pack.  The tiled kernels
// give such a problem a handful of CTAs whose threads each run a long chain
// of dependent global loads, so the launch is latency-bound.  Here a target
// has k warps (1 to 16, chosen on the host so that the CTAs of 16 warps fill
// the SMs).  A CTA builds the source records in shared memory from
// the raw nodes (build_record, a tile at a time), the lanes of a target's
// warps take every 32k-th record of the tile, and one correction entry each
// (fetched before the pair loop, so that its latency hides behind it).  The
// lanes' sums are reduced over the warp, the warps' in a fixed order, and lane
// 0 of the target's first warp applies the kernel constant to the pair sum, adds
// the correction sum and alpha/beta.  The step is pair_step's (the one-sided
// kernel's arithmetic).
//
// What bounds it is the launch and two L2 latencies.  An earlier form gave a
// cluster of CTAs 32 targets, one per lane, and added the slices' sums through
// distributed shared memory.  Back to back products (start of a kernel seen in
// steps of about 1 us): 2D DL, 1,000 nodes 8.19 -> 7.17 us, 2D SL 13.3 -> 10.2,
// Helmholtz SL, 768 nodes 10.2 -> 8.2; eight warps per CTA 8.19, 12.3 and 8.2.
// ---------------------------------------------------------------------------
constexpr int kSmallWarps = 16;

struct SmallSources {
  const double *xs, *ns, *w, *sigma;
  double2 c1, c2;
};

// Records per staged tile: one or two per thread, up to 40 KB.
template <int N>
constexpr int small_tile() {
  return N <= 4 ? 1024 : 512;
}

template <int PDE, int KIND, int DIM>
__global__ void __launch_bounds__(32 * kSmallWarps) pair_small_kernel(int64_t m, int64_t n, const double* tc,
                                                                      const double* tn, SmallSources src,
                                                                      double k, double kT, double delta,
                                                                      const double2* expi, int lk, EpiArgs e) {
  using RC = Rec<PDE, KIND, DIM, double>;
  constexpr bool CPLX = RC::cplx;
  constexpr int NT = 32 * kSmallWarps;
  constexpr int TILE = small_tile<RC::n>();
  extern __shared__ __align__(16) double recs[];  // TILE records
  __shared__ double4 sums[kSmallWarps];
  __shared__ double2 tab[CPLX ? kExpiTable : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kw = 1 << lk, sub = warp & (kw - 1);  // warps of a target; this one
  const int64_t i = (int64_t)blockIdx.x * (kSmallWarps >> lk) + (warp >> lk);
  const bool live = i < m;
  if (CPLX)
    for (int q = threadIdx.x; q < kExpiTable; q += NT) tab[q] = expi[q];
  Target<double, DIM, RC::tnormal> t;
  int64_t p = 0, p1 = 0;  // this lane's next correction entry, row end
  double2 yo = make_double2(0.0, 0.0), cv = yo;
  int32_t cj = -1;
  if (live) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) t.x[c] = tc[DIM * i + c];
    if constexpr (RC::tnormal) {
#pragma unroll
      for (int c = 0; c < DIM; ++c) t.n[c] = tn[DIM * i + c];
    }
    if (e.rowptr) {
      p = e.rowptr[i] + sub * 32 + lane;
      p1 = e.rowptr[i + 1];
    }
    if (lane == 0 && sub == 0 && !e.beta_zero) yo = epilogue_y_old<CPLX>(e, i);
  }
  auto entry = [&]() {  // value and column of entry p
    cj = e.col[p];
    cv = CPLX ? reinterpret_cast<const double2*>(e.val)[p] : make_double2(e.val[p], 0.0);
  };
  double ar = 0.0, ai = 0.0, cr = 0.0, ci = 0.0;
  // A thread's records of a tile: all loads before the first store to shared
  // memory (which the compiler may not move them across), the next tile's
  // before the pairs of this one.
  constexpr int U = TILE / NT;
  double rec[U][RC::n];
  auto fetch = [&](int64_t base) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      build_record<PDE, KIND, DIM, double>(base + threadIdx.x + u * NT, n, src.xs, src.ns, src.w, src.sigma, src.c1,
                                           src.c2, rec[u]);
  };
  fetch(0);
  for (int64_t base = 0; base < n; base += TILE) {
    const int cnt = (int)(n - base < TILE ? n - base : TILE);
    if (base) __syncthreads();  // the previous tile is consumed
#pragma unroll
    for (int u = 0; u < U; ++u) {
      double2* o = reinterpret_cast<double2*>(recs + (threadIdx.x + u * NT) * RC::n);
#pragma unroll
      for (int c = 0; c < RC::n / 2; ++c) o[c] = make_double2(rec[u][2 * c], rec[u][2 * c + 1]);
    }
    if (base == 0 && p < p1) entry();
    __syncthreads();
    if (base + TILE < n) fetch(base + TILE);
    if (live) {
      constexpr int UNROLL = PDE == LAPLACE && KIND == SL && DIM == 2 ? 1 : 4;  // (a log is long enough)
#pragma unroll UNROLL
      for (int q = sub * 32 + lane; q < cnt; q += 32 * kw)
        pair_step<PDE, KIND, DIM, double>(t, recs + q * RC::n, kT, delta, k, tab, ar, ai);
    }
  }
  while (cj >= 0) {
    if (CPLX) {
      const double2 xv = reinterpret_cast<const double2*>(e.x)[cj];
      cr = fma(cv.x, xv.x, fma(-cv.y, xv.y, cr));
      ci = fma(cv.x, xv.y, fma(cv.y, xv.x, ci));
    } else {
      cr = fma(cv.x, e.x[cj], cr);
    }
    cj = -1;
    p += 32 * kw;
    if (p < p1) entry();
  }
  double4 acc = make_double4(warp_sum(ar), CPLX ? warp_sum(ai) : 0.0, warp_sum(cr), CPLX ? warp_sum(ci) : 0.0);
  if (kw > 1) {
    if (lane == 0) sums[warp] = acc;
    __syncthreads();
    if (sub == 0)
      for (int w = 1; w < kw; ++w) {
        const double4 v = sums[warp + w];
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
      }
  }
  if (live && lane == 0 && sub == 0) {
    const double sc = e.rowscale ? e.scale * e.rowscale[i] : e.scale;
    epilogue_store<CPLX>(e, i, fma(acc.x, sc, acc.z), fma(acc.y, sc, acc.w), yo);
  }
}

// ---------------------------------------------------------------------------
// Symmetric form for square operators (the target set is the source set),// ---------------------------------------------------------------------------
// Symmetric form for square operators (the target set is the source set),
// every kernel: single layer, double layer, combined field (3D), adjoint
// double layer and hypersingular, in 3D and for the 2D Laplace kernels.
//
// Every kernel value of an unordered pair {a, b} serves both products:
//   SL: G(x_a, x_b) = G(x_b, x_a);
//   DL: K(x_a, x_b) p_b = d(r.p_b) and K(x_b, x_a) p_a = -d(r.p_a) with the
//       same radial factor d (r = x_a - x_b, p the packed dipoles w sigma n);
//   ADL and HS: see pair_sym_step;
// so the distance, the reciprocal square root and the phase are computed
// once per unordered pair.  Nodes are cut into blocks of BT = 128*TPT; a CTA
// takes one work item (row block I, source blocks J0 <= J < J1, J >= I):
// its threads hold the targets of block I (coordinates and their own packed
// charge/dipole), source tiles of the blocks J stream through shared memory
// as in pair_forward.  For J == I every ordered pair is evaluated (the
// forward step).  For J > I the row sums go to the target registers and the
// column sums of each source are reduced over the CTA (warp shuffles, then
// the four warps in a fixed order) and stored in zpart[I][j].  The epilogue
// adds, for node i of block B, the row partials of the items of row B and
// zpart[I][i] for I < B: a fixed order, so the result is deterministic.
// ---------------------------------------------------------------------------
struct SymArgs {
  int64_t npad;           // packed records: nb * BT (zero charges past n)
  const int32_t* items;   // (I, J0, J1) per CTA
  const int32_t* ids;     // row-partial slot of each CTA's item (NULL: the CTA index)
  int sub;                // CTAs per item: an equal part of its (one) source block each
  const void* packed;
  void* ypart;            // [item][BT]
  void* zpart;            // [nb][zld]: node j of the panel's columns at j - zcol0
  int64_t zld, zcol0;     // one panel: npad and 0
  double k, kT, delta;
  const void* expi;
  int* err;
};

// Records of the symmetric form.  SL, DL and CF use the layouts of Rec.  The
// adjoint double layer and the hypersingular kernel take the normal of the
// target, so both ends of a pair need their normal and their charge:
//   x [DIM] | n [DIM] | q            (Laplace; 3D: 8 elements with one pad,
//                                     2D: 6 (FP64) or 8 (FP32))
//   x y z | n_x n_y n_z | qr qi      (Helmholtz: 8 elements)
// with q = w sigma; padded to a multiple of 16 bytes.
template <int PDE, int KIND, int DIM, class R>
struct SymRec {
  static constexpr bool normal = (KIND == ADL || KIND == HS);
  static constexpr bool cplx = (PDE == HELMHOLTZ);
  static constexpr int align = 16 / sizeof(R);
  static constexpr int nused = 2 * DIM + (cplx ? 2 : 1);
  static constexpr int used = normal ? nused : Rec<PDE, KIND, DIM, R>::used;
  static constexpr int n = normal ? (nused + align - 1) / align * align : Rec<PDE, KIND, DIM, R>::n;
};

template <int PDE, int DIM, class R>
__global__ void pack_sym_normal(int64_t n, int64_t npad, const double* __restrict__ xs,
                                const double* __restrict__ ns, const double* __restrict__ w,
                                const double* __restrict__ sigma, R* __restrict__ out) {
  constexpr int NR = SymRec<PDE, HS, DIM, R>::n;
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (j >= npad) return;
  R rec[NR];
#pragma unroll
  for (int c = 0; c < NR; ++c) rec[c] = R(0);
  if (j < n) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      rec[c] = R(xs[DIM * j + c]);
      rec[DIM + c] = R(ns[DIM * j + c]);
    }
    const double wj = w[j];
    if (PDE == HELMHOLTZ) {
      rec[2 * DIM] = R(wj * sigma[2 * j]);
      rec[2 * DIM + 1] = R(wj * sigma[2 * j + 1]);
    } else {
      rec[2 * DIM] = R(wj * sigma[j]);
    }
  }
  R* o = out + j * NR;
#pragma unroll
  for (int c = 0; c < NR; ++c) o[c] = rec[c];
}

// Both products of one unordered pair: y_t += K(x_t, x_s) c_s and
// z_s += K(x_s, x_t) c_t, with c the packed charge/dipole records of the
// target t and the source s (layouts of SymRec), r = x_t - x_s.  With COL
// false only the row product is formed (the diagonal blocks of the
// adjoint double layer and hypersingular forms, which evaluate every ordered
// pair).
//   ADL: K(x_t, x_s) q_s = (r.n_t) f q_s and K(x_s, x_t) q_t = -(r.n_s) f q_t
//        with the same radial factor f (1/d^3; e^{ikd}(1/d - ik)/d^2);
//   HS : K(x_t, x_s) q_s = h q_s and K(x_s, x_t) q_t = h q_t with
//        h = a (r.n_t)(r.n_s) + b (n_t.n_s), a and b functions of d alone
//        (Laplace: a = -3/d^5, b = 1/d^3), so h is symmetric in the pair.
// 2D Laplace (kernel constants in the epilogue as in pair_step):
//   SL : log(d^2), symmetric;   DL : (r.p)/d^2, column -(r.p_t)/d^2;
//   ADL: (r.n_t) q/d^2, column -(r.n_s) q_t/d^2;
//   HS : h = (n_t.n_s - 2 (r.n_t)(r.n_s)/d^2)/d^2, symmetric.
template <int KIND, class R, bool COL>
__device__ __forceinline__ void pair_sym_step_2d(const R* __restrict__ t, const R* __restrict__ s, R& ar,
                                                 R& zr) {
  using M = MathOps<R>;
  const R r0 = t[0] - s[0], r1 = t[1] - s[1];
  const R d2 = fma(r1, r1, r0 * r0);
  const bool keep = M::keep(d2);
  if (KIND == SL) {
    const R l = keep ? M::lg(d2) : R(0);
    ar = fma(l, s[2], ar);
    if (COL) zr = fma(l, t[2], zr);
    return;
  }
  const R id2 = keep ? M::rcp(d2) : R(0);
  if (KIND == DL) {
    ar = fma(fma(r1, s[3], r0 * s[2]), id2, ar);
    if (COL) zr = fma(-fma(r1, t[3], r0 * t[2]), id2, zr);
  } else if (KIND == ADL) {
    ar = fma(fma(r1, t[3], r0 * t[2]) * id2, s[4], ar);
    if (COL) zr = fma(-fma(r1, s[3], r0 * s[2]) * id2, t[4], zr);
  } else if (KIND == HS) {
    const R rnt = fma(r1, t[3], r0 * t[2]), rns = fma(r1, s[3], r0 * s[2]);
    const R nn = fma(t[3], s[3], t[2] * s[2]);
    const R h = fma(R(-2) * rnt * rns, id2, nn) * id2;
    ar = fma(h, s[4], ar);
    if (COL) zr = fma(h, t[4], zr);
  }
}

template <int PDE, int KIND, int DIM, class R, bool COL = true>
__device__ __forceinline__ void pair_sym_step(const R* __restrict__ t, const R* __restrict__ s, R kT, R delta, R k,
                                              const typename MathOps<R>::R2* __restrict__ tab, R& ar, R& ai,
                                              R& zr, R& zi) {
  if constexpr (DIM == 2) {
    pair_sym_step_2d<KIND, R, COL>(t, s, ar, zr);
    return;
  }
  using M = MathOps<R>;
  const R r0 = t[0] - s[0], r1 = t[1] - s[1], r2 = t[2] - s[2];
  const R d2 = fma(r2, r2, fma(r1, r1, r0 * r0));
  const bool keep = M::keep(d2);
  if (KIND == ADL || KIND == HS) {
    const R rnt = fma(r2, t[5], fma(r1, t[4], r0 * t[3]));
    const R rns = COL || KIND == HS ? fma(r2, s[5], fma(r1, s[4], r0 * s[3])) : R(0);
    if (PDE == LAPLACE) {
      if (KIND == ADL) {
        const R ri3 = keep ? M::rsq3(d2) : R(0);
        ar = fma(rnt * ri3, s[6], ar);
        if (COL) zr = fma(-rns * ri3, t[6], zr);
      } else {
        const R nn = fma(t[5], s[5], fma(t[4], s[4], t[3] * s[3]));
        const R ri = keep ? M::rsq(d2) : R(0);
        const R id2 = ri * ri;
        const R h = fma(R(-3) * rnt * rns, id2, nn) * (id2 * ri);
        ar = fma(h, s[6], ar);
        if (COL) zr = fma(h, t[6], zr);
      }
    } else {
      const R ri = keep ? M::rsq(d2) : R(0);
      const R d = d2 * ri;
      R sn, cs;
      expi_table_eval(d, kT, tab, delta, cs, sn);
      const R id2 = ri * ri;
      R hr, hi, gr = R(0), gi = R(0);  // row factor h, column factor g
      if (KIND == ADL) {
        const R er = fma(cs, ri, k * sn), ei = fma(sn, ri, -k * cs);  // e^{ikd}(1/d - ik)
        const R br = er * id2, bi = ei * id2;
        hr = br * rnt;
        hi = bi * rnt;
        if (COL) {
          gr = -br * rns;
          gi = -bi * rns;
        }
      } else {
        // h = b (n_t.n_s) + a (r.n_t)(r.n_s) with b = e^{ikd}(1/d - ik)/d^2 and
        // a = e^{ikd}(k^2 d^2 - 3 + 3ikd)/d^5, i.e. h = e^{ikd} W with the
        // bracket W = (1/d - ik) p + (k^2 d^2 - 3 + 3ikd) s formed in real
        // arithmetic from p = (n_t.n_s)/d^2 and s = (r.n_t)(r.n_s)/d^5
        const R nn = fma(t[5], s[5], fma(t[4], s[4], t[3] * s[3]));
        const R kd = k * d;
        const R fr = fma(kd, kd, R(-3)), fi = R(3) * kd;
        const R p = nn * id2;
        const R s5 = (rnt * rns) * (id2 * id2 * ri);
        const R wr = fma(ri, p, fr * s5), wi = fma(-k, p, fi * s5);
        hr = fma(cs, wr, -sn * wi);
        hi = fma(cs, wi, sn * wr);
        gr = hr;
        gi = hi;
      }
      ar = fma(hr, s[6], fma(-hi, s[7], ar));
      ai = fma(hr, s[7], fma(hi, s[6], ai));
      if (COL) {
        zr = fma(gr, t[6], fma(-gi, t[7], zr));
        zi = fma(gr, t[7], fma(gi, t[6], zi));
      }
    }
    return;
  }
  if (PDE == LAPLACE) {
    if (KIND == SL) {
      const R ri = keep ? M::rsq(d2) : R(0);
      ar = fma(ri, s[3], ar);
      zr = fma(ri, t[3], zr);
    } else {
      const R rs = fma(r2, s[5], fma(r1, s[4], r0 * s[3]));
      const R rt = fma(r2, t[5], fma(r1, t[4], r0 * t[3]));
      if (KIND == DL) {
        const R ri3 = keep ? M::rsq3(d2) : R(0);
        ar = fma(rs, ri3, ar);
        zr = fma(-rt, ri3, zr);
      } else {  // CF: charge after the dipole
        const R ri = keep ? M::rsq(d2) : R(0);
        const R ri3 = ri * ri * ri;
        ar = fma(ri, s[6], fma(rs, ri3, ar));
        zr = fma(ri, t[6], fma(-rt, ri3, zr));
      }
    }
  } else {
    const R ri = keep ? M::rsq(d2) : R(0);
    R sn, cs;
    expi_table_eval(d2 * ri, kT, tab, delta, cs, sn);
    if (KIND == SL) {
      const R gr = ri * cs, gi = ri * sn;
      ar = fma(gr, s[3], fma(-gi, s[4], ar));
      ai = fma(gr, s[4], fma(gi, s[3], ai));
      zr = fma(gr, t[3], fma(-gi, t[4], zr));
      zi = fma(gr, t[4], fma(gi, t[3], zi));
    } else {  // dipole Re [3..5], Im [6..8]; CF: charge [9], [10]
      const R er = fma(cs, ri, k * sn), ei = fma(sn, ri, -k * cs);
      const R id2 = ri * ri;
      const R gr = er * id2, gi = ei * id2;
      const R A = fma(r2, s[5], fma(r1, s[4], r0 * s[3])), B = fma(r2, s[8], fma(r1, s[7], r0 * s[6]));
      const R At = fma(r2, t[5], fma(r1, t[4], r0 * t[3])), Bt = fma(r2, t[8], fma(r1, t[7], r0 * t[6]));
      ar = fma(gr, A, fma(-gi, B, ar));
      ai = fma(gr, B, fma(gi, A, ai));
      zr = fma(-gr, At, fma(gi, Bt, zr));
      zi = fma(-gr, Bt, fma(-gi, At, zi));
      if (KIND == CF) {
        const R hr = cs * ri, hi = sn * ri;
        ar = fma(hr, s[9], fma(-hi, s[10], ar));
        ai = fma(hr, s[10], fma(hi, s[9], ai));
        zr = fma(hr, t[9], fma(-hi, t[10], zr));
        zi = fma(hr, t[10], fma(hi, t[9], zi));
      }
    }
  }
}

// Warp sums of four values v[0..3] (one per source), reduce-scattered: lanes
// 0, 8, 16, 24 return the totals of v[0], v[1], v[2], v[3].  Levels 16 and 8
// exchange halves of the set instead of reducing every value over all five
// levels: 6 adds and 6 shuffles for four sums instead of 20 each.
template <class R>
__device__ __forceinline__ R warp_sum4(const R (&v)[4], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8;
  R k0 = b4 ? v[2] : v[0], k1 = b4 ? v[3] : v[1];
  k0 += __shfl_xor_sync(0xffffffffu, b4 ? v[0] : v[2], 16);
  k1 += __shfl_xor_sync(0xffffffffu, b4 ? v[1] : v[3], 16);
  R k = b3 ? k1 : k0;
  k += __shfl_xor_sync(0xffffffffu, b3 ? k0 : k1, 8);
  k += __shfl_xor_sync(0xffffffffu, k, 4);
  k += __shfl_xor_sync(0xffffffffu, k, 2);
  k += __shfl_xor_sync(0xffffffffu, k, 1);
  return k;
}

__device__ __forceinline__ void put_partial(double* p, double r, double) { *p = r; }
__device__ __forceinline__ void put_partial(double2* p, double r, double i) { *p = make_double2(r, i); }
__device__ __forceinline__ void put_partial(float2* p, float r, float) { *p = make_float2(r, 0.f); }
__device__ __forceinline__ void put_partial(float4* p, float r, float i) { *p = make_float4(r, 0.f, i, 0.f); }

// SUB: several CTAs share an item's source block (a.sub > 1).  Without it the
// tile length is a constant: made a variable it cost 4% at 62,208 nodes, and
// up to 38 registers.
template <int PDE, int KIND, int DIM, class R, int TILE, int TPT, bool SUB>
__global__ void __launch_bounds__(kBlock, (symm_min_ctas<PDE, KIND, DIM, R>())) pair_symm(SymArgs a) {
  using RC = SymRec<PDE, KIND, DIM, R>;
  constexpr bool CPLX = RC::cplx;
  using P = typename PartialT<R, CPLX>::T;
  using R2 = typename MathOps<R>::R2;
  constexpr int BT = kBlock * TPT;
  static_assert(BT % TILE == 0, "whole source tiles per node block");
  constexpr int TPB = BT / TILE;
  constexpr int NU = RC::used;
  constexpr int kWarps = kBlock / 32;
  constexpr uint32_t kStageBytes = TILE * RC::n * sizeof(R);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* stage0 = reinterpret_cast<R*>(smem_raw);
  R* stage1 = reinterpret_cast<R*>(smem_raw + kStageBytes);
  R2* tab = reinterpret_cast<R2*>(smem_raw + 2 * kStageBytes);  // Helmholtz only
  R* zsm = reinterpret_cast<R*>(smem_raw + 2 * kStageBytes + (CPLX ? kExpiTable * sizeof(R2) : 0));
  __shared__ __align__(8) uint64_t full[2], tab_full;
  constexpr bool TMA_TAB = SUB && CPLX && sizeof(R) == 8;  // (FP32 takes the hardware sine and cosine)

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // SUB: this CTA takes part `part` of the item's one source block
  const int item = SUB ? blockIdx.x / a.sub : blockIdx.x, part = SUB ? blockIdx.x % a.sub : 0;
  const int I = a.items[3 * item], J0 = a.items[3 * item + 1], J1 = a.items[3 * item + 2];
  const int ps = SUB ? BT / a.sub : 0;                           // sources of a part
  const int64_t j0 = SUB ? (int64_t)J0 * BT + part * ps : 0;     // tile t starts at source j0 + t * TILE
  auto bytes = [&](int64_t t) {
    return (SUB ? (uint32_t)min((int64_t)TILE, ps - t * TILE) : (uint32_t)TILE) * (uint32_t)(kStageBytes / TILE);
  };
  const R* src = static_cast<const R*>(a.packed);
  pdl_trigger();
  if (TMA_TAB && tid == 0) {  // the table's copy does not wait for the kernel before
    mbar_init(&tab_full, 1);
    mbar_fence_init();
    mbar_arrive_expect_tx(&tab_full, kExpiTable * sizeof(R2));
    bulk_copy_g2s(tab, a.expi, kExpiTable * sizeof(R2), &tab_full);
  }
  pdl_wait();  // the packed records; the partials of the product before are consumed
  R tg[TPT][NU];
  Acc<R, CPLX> acc[TPT];
#pragma unroll
  for (int u = 0; u < TPT; ++u) {
    const int64_t i = (int64_t)I * BT + u * kBlock + tid;
#pragma unroll
    for (int c = 0; c < NU; ++c) tg[u][c] = src[i * RC::n + c];
  }
  const R k = R(a.k), kT = R(a.kT), delta = R(a.delta);
  if (CPLX && !TMA_TAB) {
    const R2* g = static_cast<const R2*>(a.expi);
    for (int q = tid; q < kExpiTable; q += kBlock) tab[q] = g[q];
  }
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  const int64_t t0 = SUB ? 0 : (int64_t)J0 * TPB, t1 = SUB ? (ps + TILE - 1) / TILE : (int64_t)J1 * TPB;
  int64_t issued = t0;
  if (tid == 0) {
    for (int s = 0; s < 2 && issued < t1; ++s, ++issued) {
      mbar_arrive_expect_tx(&full[s], bytes(issued));
      bulk_copy_g2s(s ? stage1 : stage0, src + (j0 + issued * TILE) * RC::n, bytes(issued), &full[s]);
    }
  }
  for (int64_t t = t0; t < t1; ++t) {
    const int st = (int)((t - t0) & 1);
    const uint32_t parity = (uint32_t)(((t - t0) >> 1) & 1);
    bool ok = mbar_wait_bounded(&full[st], parity);
    if (TMA_TAB && t == t0) ok = mbar_wait_bounded(&tab_full, 0) && ok;
    if (!__syncthreads_and(ok)) {
      if (tid == 0) {
        atomicExch(a.err, kErrWaitTimeout);
        if (TMA_TAB) mbar_wait_bounded(&tab_full, 0);
        for (int64_t q = t + 1; q < issued; ++q)
          mbar_wait_bounded(&full[(q - t0) & 1], (uint32_t)(((q - t0) >> 1) & 1));
      }
      return;
    }
    const R* sp = st ? stage1 : stage0;
    const bool diag = SUB ? J0 == I : t / TPB == I;
    const int cnt = SUB ? (int)min((int64_t)TILE, ps - t * TILE) : TILE;
    R* zb = zsm + st * (kWarps * TILE * 2);
    if (diag) {
#pragma unroll 1
      for (int g = 0; g < cnt; g += kGroup) {
#pragma unroll(SUB ? 8 / TPT : 2)
        for (int s = 0; s < kGroup; ++s) {
          const R* rec = sp + (g + s) * RC::n;
#pragma unroll
          for (int u = 0; u < TPT; ++u) {
            if constexpr (RC::normal) {
              R unused_r = R(0), unused_i = R(0);  // the column half is not formed
              pair_sym_step<PDE, KIND, DIM, R, false>(tg[u], rec, kT, delta, k, tab, acc[u].gr(), acc[u].gi(),
                                                      unused_r, unused_i);
            } else {
              Target<R, DIM, false> tt;
#pragma unroll
              for (int c = 0; c < DIM; ++c) tt.x[c] = tg[u][c];
              pair_step<PDE, KIND, DIM, R>(tt, rec, kT, delta, k, tab, acc[u].gr(), acc[u].gi());
            }
          }
        }
#pragma unroll
        for (int u = 0; u < TPT; ++u) acc[u].fold();
      }
    } else {
#pragma unroll 1
      for (int g = 0; g < cnt; g += kGroup) {
#pragma unroll 1
        for (int s = 0; s < kGroup; s += 4) {
          R zr[4], zi[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const R* rec = sp + (g + s + v) * RC::n;
            zr[v] = zi[v] = R(0);
#pragma unroll
            for (int u = 0; u < TPT; ++u)
              pair_sym_step<PDE, KIND, DIM, R>(tg[u], rec, kT, delta, k, tab, acc[u].gr(), acc[u].gi(), zr[v],
                                               zi[v]);
          }
          const R sr = warp_sum4(zr, lane);
          const R si = CPLX ? warp_sum4(zi, lane) : R(0);
          if ((lane & 7) == 0) {
            const int v = lane >> 3;
            zb[(warp * TILE + g + s + v) * 2] = sr;
            zb[(warp * TILE + g + s + v) * 2 + 1] = si;
          }
        }
#pragma unroll
        for (int u = 0; u < TPT; ++u) acc[u].fold();
      }
    }
    __syncthreads();  // the stage is read and this tile's column sums are in zb
    if (!diag) {
      P* zp = static_cast<P*>(a.zpart) + (int64_t)I * a.zld + (j0 + t * TILE - a.zcol0);
      for (int s = tid; s < cnt; s += kBlock) {
        R vr = zb[s * 2], vi = zb[s * 2 + 1];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) {
          vr += zb[(w * TILE + s) * 2];
          vi += zb[(w * TILE + s) * 2 + 1];
        }
        put_partial(zp + s, vr, vi);
      }
    }
    if (tid == 0 && issued < t1) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[st], bytes(issued));
      bulk_copy_g2s(st ? stage1 : stage0, src + (j0 + issued * TILE) * RC::n, bytes(issued), &full[st]);
      ++issued;
    }
  }
  P* out = static_cast<P*>(a.ypart) + (int64_t)((a.ids ? a.ids[item] : item) * (SUB ? a.sub : 1) + part) * BT;
#pragma unroll
  for (int u = 0; u < TPT; ++u) store_partial(out + u * kBlock + tid, acc[u]);
}

// ---------------------------------------------------------------------------
// Paired-FP32 form of the symmetric kernel for the FP32C Laplace single
// layer, double layer and combined field (3D).  The FP32 kernels are bound by
// instruction issue, not by the FP32 pipe; sm_100 issues two FP32 lanes per
// instruction (__fadd2_rn, __fmul2_rn, __ffma2_rn).  Each thread holds its
// targets in pairs (u, u + 1) as float2, and the records carry every value
// twice (x x y y z z | p_x p_x p_y p_y p_z p_z | q q), so one 16-byte shared
// load yields two ready operand pairs.  Per lane the arithmetic is that of
// pair_sym_step (the reciprocal square root and the self-pair test stay per
// lane); the column sum over the thread's targets is formed per lane and the
// two lanes added, so results differ from the scalar kernel by rounding only.
// ---------------------------------------------------------------------------
template <int KIND>
struct RecX2 {
  static constexpr int vals = (KIND == SL ? 4 : KIND == DL ? 6 : 7);  // x y z [p] [q]
  static constexpr int n = (2 * vals + 3) / 4 * 4;                      // floats per record
};

template <int KIND>
__global__ void pack_sources_x2(int64_t n, int64_t npad, const double* __restrict__ xs,
                                const double* __restrict__ ns, const double* __restrict__ w,
                                const double* __restrict__ sigma, double c1, double c2,
                                float* __restrict__ out) {
  constexpr int NR = RecX2<KIND>::n;
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  pdl_trigger();
  pdl_wait();
  if (j >= npad) return;
  float v[RecX2<KIND>::vals];
#pragma unroll
  for (int c = 0; c < RecX2<KIND>::vals; ++c) v[c] = 0.f;
  if (j < n) {
    v[0] = (float)xs[3 * j];
    v[1] = (float)xs[3 * j + 1];
    v[2] = (float)xs[3 * j + 2];
    const double q = w[j] * sigma[j];
    if (KIND == SL) {
      v[3] = (float)q;
    } else {
      const double qd = KIND == CF ? c1 * q : q;
#pragma unroll
      for (int c = 0; c < 3; ++c) v[3 + c] = (float)(qd * ns[3 * j + c]);
      if (KIND == CF) v[6] = (float)(c2 * q);
    }
  }
  float* o = out + j * NR;
#pragma unroll
  for (int c = 0; c < NR; ++c) o[c] = c / 2 < RecX2<KIND>::vals ? v[c / 2] : 0.f;
}

// One source against a pair of targets: the row products into (ar.x, ar.y);
// with COL the column terms into zq (ri q_t, CF) and zd (r.p_t ri^3).
template <int KIND, bool COL>
__device__ __forceinline__ void pair_x2_step(const float2 (&t)[RecX2<KIND>::vals], const float2* __restrict__ s,
                                             float2& ar, float2& zq, float2& zd) {
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 r0 = __ffma2_rn(s[0], m1, t[0]);  // t - s, one rounding per lane
  const float2 r1 = __ffma2_rn(s[1], m1, t[1]);
  const float2 r2 = __ffma2_rn(s[2], m1, t[2]);
  const float2 d2 = __ffma2_rn(r2, r2, __ffma2_rn(r1, r1, __fmul2_rn(r0, r0)));
  float2 ri;
  ri.x = d2.x > 1.0e-28f ? rsqrt_fast(d2.x) : 0.f;
  ri.y = d2.y > 1.0e-28f ? rsqrt_fast(d2.y) : 0.f;
  if (KIND == SL) {
    ar = __ffma2_rn(ri, s[3], ar);
    if (COL) zq = __ffma2_rn(ri, t[3], zq);
    return;
  }
  const float2 ri3 = __fmul2_rn(__fmul2_rn(ri, ri), ri);
  const float2 rs = __ffma2_rn(r2, s[5], __ffma2_rn(r1, s[4], __fmul2_rn(r0, s[3])));
  if (KIND == CF) {
    ar = __ffma2_rn(ri, s[6], __ffma2_rn(rs, ri3, ar));
  } else {
    ar = __ffma2_rn(rs, ri3, ar);
  }
  if (COL) {
    const float2 rt = __ffma2_rn(r2, t[5], __ffma2_rn(r1, t[4], __fmul2_rn(r0, t[3])));
    zd = __ffma2_rn(rt, ri3, zd);
    if (KIND == CF) zq = __ffma2_rn(ri, t[6], zq);
  }
}

template <int KIND, int TPT, bool SUB>
__global__ void __launch_bounds__(kBlock) pair_symm_x2(SymArgs a) {
  constexpr int TILE = kTile32;
  constexpr int NR = RecX2<KIND>::n, NV = RecX2<KIND>::vals;
  constexpr int BT = kBlock * TPT, NP = TPT / 2;
  static_assert(TPT % 2 == 0 && BT % TILE == 0, "target pairs, whole source tiles per node block");
  constexpr int TPB = BT / TILE;
  constexpr int kWarps = kBlock / 32;
  constexpr uint32_t kStageBytes = TILE * NR * sizeof(float);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* stage0 = reinterpret_cast<float*>(smem_raw);
  float* stage1 = reinterpret_cast<float*>(smem_raw + kStageBytes);
  float* zsm = reinterpret_cast<float*>(smem_raw + 2 * kStageBytes);
  __shared__ __align__(8) uint64_t full[2];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // SUB: this CTA takes part `part` of the item's one source block
  const int item = SUB ? blockIdx.x / a.sub : blockIdx.x, part = SUB ? blockIdx.x % a.sub : 0;
  const int I = a.items[3 * item], J0 = a.items[3 * item + 1], J1 = a.items[3 * item + 2];
  const int ps = SUB ? BT / a.sub : 0;                           // sources of a part
  const int64_t j0 = SUB ? (int64_t)J0 * BT + part * ps : 0;     // tile t starts at source j0 + t * TILE
  auto bytes = [&](int64_t t) {
    return (SUB ? (uint32_t)min((int64_t)TILE, ps - t * TILE) : (uint32_t)TILE) * (uint32_t)(kStageBytes / TILE);
  };
  const float* src = static_cast<const float*>(a.packed);
  pdl_trigger();
  pdl_wait();  // the packed records; the partials of the product before are consumed
  float2 tg[NP][NV];  // (target 2p, target 2p + 1), value c
  float2 g[NP];       // group sums per lane
  float hr[TPT], lr[TPT];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int64_t i0 = (int64_t)I * BT + (2 * p) * kBlock + tid, i1 = i0 + kBlock;
#pragma unroll
    for (int c = 0; c < NV; ++c) tg[p][c] = make_float2(src[i0 * NR + 2 * c], src[i1 * NR + 2 * c]);
    g[p] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int u = 0; u < TPT; ++u) hr[u] = lr[u] = 0.f;
  auto fold = [&]() {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      two_sum_fold(hr[2 * p], lr[2 * p], g[p].x);
      two_sum_fold(hr[2 * p + 1], lr[2 * p + 1], g[p].y);
    }
  };
  if (tid == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_fence_init();
  }
  __syncthreads();
  const int64_t t0 = SUB ? 0 : (int64_t)J0 * TPB, t1 = SUB ? (ps + TILE - 1) / TILE : (int64_t)J1 * TPB;
  int64_t issued = t0;
  if (tid == 0) {
    for (int s = 0; s < 2 && issued < t1; ++s, ++issued) {
      mbar_arrive_expect_tx(&full[s], bytes(issued));
      bulk_copy_g2s(s ? stage1 : stage0, src + (j0 + issued * TILE) * NR, bytes(issued), &full[s]);
    }
  }
  for (int64_t t = t0; t < t1; ++t) {
    const int st = (int)((t - t0) & 1);
    const uint32_t parity = (uint32_t)(((t - t0) >> 1) & 1);
    const bool ok = mbar_wait_bounded(&full[st], parity);
    if (!__syncthreads_and(ok)) {
      if (tid == 0) {
        atomicExch(a.err, kErrWaitTimeout);
        for (int64_t q = t + 1; q < issued; ++q)
          mbar_wait_bounded(&full[(q - t0) & 1], (uint32_t)(((q - t0) >> 1) & 1));
      }
      return;
    }
    const float* sp = st ? stage1 : stage0;
    const bool diag = SUB ? J0 == I : t / TPB == I;
    const int cnt = SUB ? (int)min((int64_t)TILE, ps - t * TILE) : TILE;
    float* zb = zsm + st * (kWarps * TILE * 2);
    if (diag) {
#pragma unroll 1
      for (int gq = 0; gq < cnt; gq += kGroup) {
#pragma unroll 2
        for (int s = 0; s < kGroup; ++s) {
          const float2* rec = reinterpret_cast<const float2*>(sp + (gq + s) * NR);
          float2 zq = make_float2(0.f, 0.f), zd = zq;  // the column half is not formed
#pragma unroll
          for (int p = 0; p < NP; ++p) pair_x2_step<KIND, false>(tg[p], rec, g[p], zq, zd);
        }
        fold();
      }
    } else {
#pragma unroll 1
      for (int gq = 0; gq < cnt; gq += kGroup) {
#pragma unroll 1
        for (int s = 0; s < kGroup; s += 4) {
          float zr[4];
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const float2* rec = reinterpret_cast<const float2*>(sp + (gq + s + v) * NR);
            float2 zq = make_float2(0.f, 0.f), zd = make_float2(0.f, 0.f);
#pragma unroll
            for (int p = 0; p < NP; ++p) pair_x2_step<KIND, true>(tg[p], rec, g[p], zq, zd);
            // K(x_s, x_t) c_t: SL and CF ri q_t, DL and CF -(r.p_t) ri^3
            zr[v] = KIND == DL ? -(zd.x + zd.y) : (KIND == SL ? zq.x + zq.y : (zq.x + zq.y) - (zd.x + zd.y));
          }
          const float sr = warp_sum4(zr, lane);
          if ((lane & 7) == 0) {
            const int v = lane >> 3;
            zb[(warp * TILE + gq + s + v) * 2] = sr;
            zb[(warp * TILE + gq + s + v) * 2 + 1] = 0.f;
          }
        }
        fold();
      }
    }
    __syncthreads();  // the stage is read and this tile's column sums are in zb
    if (!diag) {
      float2* zp = static_cast<float2*>(a.zpart) + (int64_t)I * a.zld + (j0 + t * TILE - a.zcol0);
      for (int s = tid; s < cnt; s += kBlock) {
        float vr = zb[s * 2];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) vr += zb[(w * TILE + s) * 2];
        zp[s] = make_float2(vr, 0.f);
      }
    }
    if (tid == 0 && issued < t1) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[st], bytes(issued));
      bulk_copy_g2s(st ? stage1 : stage0, src + (j0 + issued * TILE) * NR, bytes(issued), &full[st]);
      ++issued;
    }
  }
  float2* out = static_cast<float2*>(a.ypart) + (int64_t)((a.ids ? a.ids[item] : item) * (SUB ? a.sub : 1) + part) * BT;
#pragma unroll
  for (int u = 0; u < TPT; ++u) out[u * kBlock + tid] = make_float2(hr[u], lr[u]);
}

// Row sums of the symmetric form: the item partials of row block B and the
// column partials of the row blocks above.
// Running sums over panels: for node i of row block B (B < the panel's
// rows), acc[i] += the panel's row partials of B's items (in order), then,
// when B is one of the panel's source blocks, the column partials
// zpart[r][i - col0*bt] of the row blocks r < B.
struct SymFold {
  int64_t m;
  int bt;
  const int32_t* rowptr;
  const int32_t* rowitems;
  const void* ypart;
  const void* zpart;
  int64_t zld;
  int col0, ncols;
  void* acc;
};

// Four threads per node: slice s sums the column partials of the row blocks
// r = s, s + 4, ...; the slices are added in a fixed order (deterministic).
constexpr int kFoldNodes = 64, kFoldSlices = 4;

template <class P, bool CPLX>
__global__ void __launch_bounds__(kFoldNodes * kFoldSlices) pair_symm_fold_kernel(SymFold f) {
  __shared__ double2 part[kFoldSlices][kFoldNodes];
  const int tn = threadIdx.x % kFoldNodes, sl = threadIdx.x / kFoldNodes;
  const int64_t i = blockIdx.x * (int64_t)kFoldNodes + tn;
  const bool live = i < f.m;
  const int B = live ? (int)(i / f.bt) : 0, il = live ? (int)(i % f.bt) : 0;
  const P* yp = static_cast<const P*>(f.ypart);
  const P* zp = static_cast<const P*>(f.zpart);
  double2 c = make_double2(0.0, 0.0);
  if (live && B >= f.col0 && B < f.col0 + f.ncols) {
    const int64_t jl = i - (int64_t)f.col0 * f.bt;
    for (int r = sl; r < B; r += kFoldSlices) {
      const double2 v = load_partial(zp + (int64_t)r * f.zld + jl);
      c.x += v.x;
      c.y += v.y;
    }
  }
  part[sl][tn] = c;
  __syncthreads();
  if (sl != 0 || !live) return;
  double sr = 0.0, si = 0.0;
  if (CPLX) {
    const double2 v = static_cast<const double2*>(f.acc)[i];
    sr = v.x;
    si = v.y;
  } else {
    sr = static_cast<const double*>(f.acc)[i];
  }
  for (int q = f.rowptr[B]; q < f.rowptr[B + 1]; ++q) {
    const double2 v = load_partial(yp + (int64_t)f.rowitems[q] * f.bt + il);
    sr += v.x;
    si += v.y;
  }
  sr += (part[0][tn].x + part[1][tn].x) + (part[2][tn].x + part[3][tn].x);
  si += (part[0][tn].y + part[1][tn].y) + (part[2][tn].y + part[3][tn].y);
  if (CPLX)
    static_cast<double2*>(f.acc)[i] = make_double2(sr, si);
  else
    static_cast<double*>(f.acc)[i] = sr;
}

struct SymEpi {
  int64_t npad;
  int bt, lsub;             // block, log2 of the slots per item
  const int32_t* rowptr;    // nb + 1
  const int32_t* rowitems;  // items of each row block
  const void* zpart;
};

// Row i of the product.  Eight threads per node, each summing every eighth
// of its partials (the slots of its block's items, then the column partials
// of the blocks above) and of its correction row's entries; the eight sums
// are added in a fixed order.  One thread per node summed them one after
// another, with 12 blocks of 256 threads at 3,072 nodes.
constexpr int kEpiNodes = 32, kEpiSlices = 8;

template <class P, bool CPLX>
__global__ void __launch_bounds__(kEpiNodes * kEpiSlices) pair_symm_epilogue_kernel(EpiArgs e, SymEpi s) {
  __shared__ double4 part[kEpiSlices][kEpiNodes];
  __shared__ int32_t list[kEpiNodes * kEpiSlices];
  const int tn = threadIdx.x % kEpiNodes, sl = threadIdx.x / kEpiNodes;
  const int64_t i0 = blockIdx.x * (int64_t)kEpiNodes, i = i0 + tn;
  const bool live = i < e.m;
  pdl_trigger();
  pdl_wait();
  double4 c = make_double4(0.0, 0.0, 0.0, 0.0);  // pair sum, correction sum
  if (live && e.rowptr) {
    for (int64_t p = e.rowptr[i] + sl, p1 = e.rowptr[i + 1]; p < p1; p += kEpiSlices) {
      const int32_t j = e.col[p];
      if (CPLX) {
        const double2 v = reinterpret_cast<const double2*>(e.val)[p];
        const double2 xv = reinterpret_cast<const double2*>(e.x)[j];
        c.z = fma(v.x, xv.x, fma(-v.y, xv.y, c.z));
        c.w = fma(v.x, xv.y, fma(v.y, xv.x, c.w));
      } else {
        c.z = fma(e.val[p], e.x[j], c.z);
      }
    }
  }
  // the nodes of a CTA lie in one row block
  const int B = (int)(i0 / s.bt), il = (int)(i - (int64_t)B * s.bt);
  const P* yp = static_cast<const P*>(e.partial) + il;
  const P* zp = static_cast<const P*>(s.zpart) + i;
  const int q0 = s.rowptr[B], q1 = s.rowptr[B + 1];
  for (int qc = q0; qc < q1; qc += kEpiNodes * kEpiSlices) {
    const int cnt = min(q1 - qc, kEpiNodes * kEpiSlices);
    __syncthreads();
    if ((int)threadIdx.x < cnt) list[threadIdx.x] = s.rowitems[qc + threadIdx.x];
    __syncthreads();
    if (live) {
#pragma unroll 4
      for (int q = sl; q < cnt << s.lsub; q += kEpiSlices) {
        const int64_t slot = ((int64_t)list[q >> s.lsub] << s.lsub) + (q & ((1 << s.lsub) - 1));
        const double2 v = load_partial(yp + slot * s.bt);
        c.x += v.x;
        c.y += v.y;
      }
    }
  }
  if (live) {
#pragma unroll 4
    for (int r = sl; r < B; r += kEpiSlices) {
      const double2 v = load_partial(zp + (int64_t)r * s.npad);
      c.x += v.x;
      c.y += v.y;
    }
  }
  part[sl][tn] = c;
  __syncthreads();
  if (sl != 0 || i >= e.m) return;
#pragma unroll
  for (int q = 1; q < kEpiSlices; ++q) {
    const double4 v = part[q][tn];
    c.x += v.x;
    c.y += v.y;
    c.z += v.z;
    c.w += v.w;
  }
  const double sc = e.rowscale ? e.scale * e.rowscale[i] : e.scale;
  epilogue_store<CPLX>(e, i, fma(c.x, sc, c.z), fma(c.y, sc, c.w),
                       e.beta_zero ? make_double2(0.0, 0.0) : epilogue_y_old<CPLX>(e, i));
}

// ---------------------------------------------------------------------------
// Dense assembly out[i + m*j] = K(x_i, y_j) w_j (column-major).
// ---------------------------------------------------------------------------
template <int PDE, int KIND, int DIM>
__global__ void assemble_kernel(int64_t m, int64_t n, const double* tc, const double* tn,
                                const double* sc, const double* sn, const double* w, double k,
                                double* out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t j = blockIdx.y;
  if (i >= m) return;
  const double2 v = kernel_value<PDE, KIND, DIM>(tc + DIM * i, tn ? tn + DIM * i : nullptr,
                                                 sc + DIM * j, sn ? sn + DIM * j : nullptr, k);
  const double wj = w[j];
  if (PDE == HELMHOLTZ) {
    reinterpret_cast<double2*>(out)[i + m * j] = make_double2(v.x * wj, v.y * wj);
  } else {
    out[i + m * j] = v.x * wj;
  }
}


// ---------------------------------------------------------------------------
// Host-side dispatch
// ---------------------------------------------------------------------------
int pair_tile(int precision) { return precision == INTI_FP32C ? kTile32 : kTile64; }

// e^{i m delta}, delta = fl(2 pi / kExpiTable), m = 0..kExpiTable-1, computed
// in x87 extended precision (m*delta is exact there) and rounded once.
static std::vector<long double> expi_host(bool sine) {
  const double delta = 2 * kPi / kExpiTable;
  std::vector<long double> v(kExpiTable);
  for (int m = 0; m < kExpiTable; ++m) {
    const long double a = (long double)m * (long double)delta;
    v[m] = sine ? sinl(a) : cosl(a);
  }
  return v;
}

const double2* expi_table_f64(inti_ctx* ctx) {
  if (!ctx->expi64.p) {
    const auto c = expi_host(false), s = expi_host(true);
    std::vector<double2> t(kExpiTable);
    for (int m = 0; m < kExpiTable; ++m) t[m] = make_double2((double)c[m], (double)s[m]);
    ctx->expi64.ensure(sizeof(double2) * kExpiTable);
    INTI_CUDA(cudaMemcpy(ctx->expi64.p, t.data(), sizeof(double2) * kExpiTable, cudaMemcpyHostToDevice));
  }
  return ctx->expi64.as<double2>();
}

const float2* expi_table_f32(inti_ctx* ctx) {
  if (!ctx->expi32.p) {
    const auto c = expi_host(false), s = expi_host(true);
    std::vector<float2> t(kExpiTable);
    for (int m = 0; m < kExpiTable; ++m) t[m] = make_float2((float)c[m], (float)s[m]);
    ctx->expi32.ensure(sizeof(float2) * kExpiTable);
    INTI_CUDA(cudaMemcpy(ctx->expi32.p, t.data(), sizeof(float2) * kExpiTable, cudaMemcpyHostToDevice));
  }
  return ctx->expi32.as<float2>();
}

template <class R>
static int rec_elems(int pde, int kind, int dim) {
  const bool dip = kind == DL || kind == HS || kind == CF;
  const bool cp = pde == HELMHOLTZ;
  const int used = dim + (cp ? 2 : 1) * ((dip ? dim : 1) + (kind == CF ? 1 : 0));
  const int al = 16 / (int)sizeof(R);
  return (used + al - 1) / al * al;
}

int pair_record_bytes(int pde, int kind, int dim, int precision) {
  return precision == INTI_FP32C ? rec_elems<float>(pde, kind, dim) * 4
                                 : rec_elems<double>(pde, kind, dim) * 8;
}

int pair_partial_bytes(int pde, int precision) {
  if (precision == INTI_FP32C) return pde == HELMHOLTZ ? 16 : 8;
  return pde == HELMHOLTZ ? 16 : 8;
}

// Kernel constant applied in the epilogue (see pair_step).
static double pair_scale(int pde, int kind, int dim) {
  const double c3 = 1.0 / (4 * kPi), c2 = 1.0 / (2 * kPi);
  if (kind == CF) return c3;  // 3D only: DL and SL share 1/(4 pi)
  if (pde == HELMHOLTZ) return kind == ADL ? -c3 : c3;
  if (dim == 2) {
    switch (kind) {
      case SL: return -1.0 / (4 * kPi);  // applied to log(d^2)
      case DL: return c2;
      case ADL: return -c2;
      default: return c2;
    }
  }
  return kind == ADL ? -c3 : c3;
}

template <class F>
static void dispatch(int pde, int kind, int dim, F&& f);

template <int PDE, int KIND, int DIM>
struct Tag {
  static constexpr int pde = PDE, kind = KIND, dim = DIM;
};

template <class F>
static void dispatch(int pde, int kind, int dim, F&& f) {
  if (pde == LAPLACE && dim == 3) {
    switch (kind) {
      case SL: return f(Tag<LAPLACE, SL, 3>());
      case DL: return f(Tag<LAPLACE, DL, 3>());
      case ADL: return f(Tag<LAPLACE, ADL, 3>());
      case HS: return f(Tag<LAPLACE, HS, 3>());
      case CF: return f(Tag<LAPLACE, CF, 3>());
    }
  } else if (pde == LAPLACE && dim == 2) {
    switch (kind) {
      case SL: return f(Tag<LAPLACE, SL, 2>());
      case DL: return f(Tag<LAPLACE, DL, 2>());
      case ADL: return f(Tag<LAPLACE, ADL, 2>());
      case HS: return f(Tag<LAPLACE, HS, 2>());
    }
  } else if (pde == HELMHOLTZ && dim == 3) {
    switch (kind) {
      case SL: return f(Tag<HELMHOLTZ, SL, 3>());
      case DL: return f(Tag<HELMHOLTZ, DL, 3>());
      case ADL: return f(Tag<HELMHOLTZ, ADL, 3>());
      case HS: return f(Tag<HELMHOLTZ, HS, 3>());
      case CF: return f(Tag<HELMHOLTZ, CF, 3>());
    }
  }
  throw Error(INTI_E_UNSUPPORTED, "unsupported operator: pde=" + std::to_string(pde) +
                                      " kernel=" + std::to_string(kind) +
                                      " dim=" + std::to_string(dim));
}

template <class T, class R, int TPT = kTPT>
static const void* fwd_kernel_ptr() {
  constexpr int TILE = std::is_same<R, float>::value ? kTile32 : kTile64;
  return reinterpret_cast<const void*>(&pair_forward<T::pde, T::kind, T::dim, R, TILE, TPT>);
}

template <class T, class R>
static size_t fwd_smem(int tile = std::is_same<R, float>::value ? kTile32 : kTile64) {
  const size_t table = T::pde == HELMHOLTZ ? (size_t)kExpiTable * 2 * sizeof(R) : 0;
  return 2 * (size_t)tile * Rec<T::pde, T::kind, T::dim, R>::n * sizeof(R) + table;
}

// Source chunks of a product of m targets and n sources.  FP64: chunks of
// whole tiles until an SM has 20 CTAs; where two targets per thread and whole
// tiles leave fewer than 10 per SM, parts of tiles (32 sources, and more chunks
// than tiles say so) until it has 12.  Equal CTAs that nearly fill one wave
// leave the SMs unevenly loaded, and few CTAs leave their latencies bare.
// Products back to back, Laplace DL: 51,894 sources x 1,000 targets with 2,
// 5.5, 11 and 22 CTAs per SM 236, 108, 72 and 70 us; 12,150 x 500 with whole
// tiles (5) 21.4, parts at 7, 10 and 20 per SM 18.7, 15.8 and 16.4; 3,456 x
// 1,000 whole tiles (3) 20.1, parts (6, 12) 14.0 and 12.1; but 3,456 x 4,096
// whole tiles (11.7) 24.5, parts 24.8.
int pair_plan_split(const inti_ctx* ctx, int pde, int kind, int dim, int precision, int64_t m,
                    int64_t n, int tpt) {
  if (tpt != 2 && tpt != 4) throw Error(INTI_E_ARG, "targets per thread must be 2 or 4");
  if (precision == INTI_FP64) {
    const int64_t blocks = (m + fwd_rows(precision, tpt) - 1) / fwd_rows(precision, tpt);
    const int64_t tiles = std::max<int64_t>(1, (n + kTile64 - 1) / kTile64);
    const int64_t units = tiles * (kTile64 / kFineTile), sms = ctx->num_sms;
    if (tpt == 2 && blocks * tiles < 10 * sms) {
      const int64_t per = std::max<int64_t>(1, (units * blocks + 6 * sms) / (12 * sms));
      const int64_t split = (units + per - 1) / per;
      if (split > tiles) return (int)split;
    }
    const int64_t per = std::max<int64_t>(1, tiles * blocks / (20 * sms));
    return (int)((tiles + per - 1) / per);
  }
  int occ = 1;
  dispatch(pde, kind, dim, [&](auto tag) {
    using T = decltype(tag);
    const void* fn = tpt == 2 ? fwd_kernel_ptr<T, float, 2>() : fwd_kernel_ptr<T, float, 4>();
    const size_t sm = fwd_smem<T, float>();
    INTI_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    INTI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBlock, sm));
  });
  occ = std::max(occ, 1);
  const int64_t tile = pair_tile(precision);
  const int64_t n_tiles = std::max<int64_t>(1, (n + tile - 1) / tile);
  const int64_t blocks = (m + fwd_rows(precision, tpt) - 1) / fwd_rows(precision, tpt);
  const int64_t slots = (int64_t)ctx->num_sms * occ;
  // Smallest split whose last wave is >= 90% full (or that reaches 8
  // waves), never more chunks than source tiles.  Up to kMaxSplit chunks:
  // few target blocks (potentials at a few thousand points) need many.
  int best = 1;
  double best_eff = -1.0;
  for (int s = 1; s <= kMaxSplit && s <= n_tiles; ++s) {
    const int64_t tps = (n_tiles + s - 1) / s;
    const int64_t eff_s = (n_tiles + tps - 1) / tps;  // chunks actually used
    const double waves = (double)(blocks * eff_s) / (double)slots;
    const double eff = waves / std::ceil(waves);
    if (eff > best_eff + 1e-9) {
      best_eff = eff;
      best = s;
    }
    if ((eff >= 0.9 && waves >= 1.0) || waves >= 8.0) {
      best = s;
      break;
    }
  }
  return best;
}

// Targets per thread: four, unless whole tiles then give an SM fewer than 12
// CTAs (Laplace DL, 12,150 sources x 2,000 targets, 10 per SM: 55.4 us with
// four, 38.6 with two; 51,894 x 1,000, 22 per SM: 70.1 and 71.2).  Transposes
// of square operators take the same rule, four from about 5,400 nodes on
// (10,800 nodes, Helmholtz DL, from host arrays: 341 -> 302 us with the slices
// and chunks above).
int pair_plan_tpt(const inti_ctx* ctx, int precision, int64_t m, int64_t n) {
  if (precision != INTI_FP64) return 4;
  const int64_t rows = fwd_rows(precision, 4);
  return (m + rows - 1) / rows * ((n + kTile64 - 1) / kTile64) < 12 * (int64_t)ctx->num_sms ? 2 : 4;
}

// Dynamic shared memory of the symmetric kernel: two source stages, the
// e^{i m delta} table, two buffers of per-warp column sums.
template <class T, class R>
static size_t symm_smem() {
  constexpr int TILE = std::is_same<R, float>::value ? kTile32 : kTile64;
  const size_t table = T::pde == HELMHOLTZ ? (size_t)kExpiTable * 2 * sizeof(R) : 0;
  return 2 * (size_t)TILE * SymRec<T::pde, T::kind, T::dim, R>::n * sizeof(R) + table +
         2 * (size_t)(kBlock / 32) * TILE * 2 * sizeof(R);
}

template <class T>
constexpr bool symm_kind() {
  return true;  // every kernel of the dispatch (3D, and 2D Laplace)
}

// FP32 Laplace SL/DL/CF in 3D run the paired-FP32 symmetric kernel.
template <class T, class R>
constexpr bool symm_x2() {
  return std::is_same<R, float>::value && T::pde == LAPLACE && T::dim == 3 &&
         (T::kind == SL || T::kind == DL || T::kind == CF);
}

template <class T>
static size_t symm_x2_smem() {
  return 2 * (size_t)kTile32 * RecX2<T::kind>::n * sizeof(float) + 2 * (size_t)(kBlock / 32) * kTile32 * 2 * sizeof(float);
}

int pair_symm_record_bytes(int pde, int kind, int dim, int precision) {
  int bytes = 0;
  dispatch(pde, kind, dim, [&](auto tag) {
    using T = decltype(tag);
    if constexpr (symm_x2<T, float>())
      bytes = precision == INTI_FP32C ? RecX2<T::kind>::n * 4 : SymRec<T::pde, T::kind, T::dim, double>::n * 8;
    else
      bytes = precision == INTI_FP32C ? SymRec<T::pde, T::kind, T::dim, float>::n * 4
                                      : SymRec<T::pde, T::kind, T::dim, double>::n * 8;
  });
  return bytes;
}

int pair_symm_block(int tpt) { return kBlock * tpt; }

void pair_symm_plan(int64_t n, int tpt, int ch, int pcols, std::vector<int32_t>& table,
                    std::vector<SymPanel>& panels, int& nb, int& nitems) {
  const int bt = pair_symm_block(tpt);
  nb = (int)std::max<int64_t>(1, (n + bt - 1) / bt);
  ch = std::max(1, ch);
  pcols = std::max(1, std::min(pcols, nb));
  table.clear();
  panels.clear();
  nitems = 0;
  for (int c0 = 0; c0 < nb; c0 += pcols) {
    const int c1 = std::min(c0 + pcols, nb);
    std::vector<std::array<int32_t, 3>> it;
    for (int I = 0; I < c1; ++I)
      for (int J0 = std::max(I, c0); J0 < c1; J0 += ch) it.push_back({I, J0, std::min(J0 + ch, c1)});
    std::stable_sort(it.begin(), it.end(), [](const std::array<int32_t, 3>& a, const std::array<int32_t, 3>& b) {
      return a[2] - a[1] > b[2] - b[1];
    });
    SymPanel P;
    P.col0 = c0;
    P.ncols = c1 - c0;
    P.rows = c1;
    P.nitems = (int)it.size();
    P.item_off = (int)table.size();  // int32 offset of the items
    P.rowptr_off = P.item_off + 3 * P.nitems;
    P.rowitems_off = P.rowptr_off + P.rows + 1;
    table.resize((size_t)P.rowitems_off + P.nitems, 0);
    int32_t* items = table.data() + P.item_off;
    int32_t* rowptr = table.data() + P.rowptr_off;
    int32_t* rowitems = table.data() + P.rowitems_off;
    for (int q = 0; q < P.nitems; ++q) {
      items[3 * q] = it[q][0];
      items[3 * q + 1] = it[q][1];
      items[3 * q + 2] = it[q][2];
      ++rowptr[it[q][0] + 1];
    }
    for (int I = 0; I < P.rows; ++I) rowptr[I + 1] += rowptr[I];
    std::vector<int32_t> fill(rowptr, rowptr + P.rows);
    for (int q = 0; q < P.nitems; ++q) rowitems[fill[it[q][0]]++] = q;
    nitems = std::max(nitems, P.nitems);
    panels.push_back(P);
  }
}

int pair_symm_default_ch(const inti_ctx* ctx, int pde, int kind, int dim, int precision, int64_t n, int tpt) {
  int occ = 1;
  dispatch(pde, kind, dim, [&](auto tag) {
    using T = decltype(tag);
    if constexpr (symm_kind<T>()) {
      const void* fn;
      size_t sm;
      if (precision == INTI_FP32C) {
        if constexpr (symm_x2<T, float>()) {
          fn = tpt == 2 ? (const void*)&pair_symm_x2<T::kind, 2, false> : (const void*)&pair_symm_x2<T::kind, 4, false>;
          sm = symm_x2_smem<T>();
        } else {
          fn = tpt == 2 ? (const void*)&pair_symm<T::pde, T::kind, T::dim, float, kTile32, 2, false>
                        : (const void*)&pair_symm<T::pde, T::kind, T::dim, float, kTile32, 4, false>;
          sm = symm_smem<T, float>();
        }
      } else {
        fn = tpt == 2 ? (const void*)&pair_symm<T::pde, T::kind, T::dim, double, kTile64, 2, false>
                      : (const void*)&pair_symm<T::pde, T::kind, T::dim, double, kTile64, 4, false>;
        sm = symm_smem<T, double>();
      }
      INTI_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      INTI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBlock, sm));
    }
  });
  occ = std::max(occ, 1);
  const int bt = pair_symm_block(tpt);
  const int64_t nb = std::max<int64_t>(1, (n + bt - 1) / bt);
  const int64_t pairs = nb * (nb + 1) / 2;         // block pairs J >= I
  const int64_t want = (int64_t)ctx->num_sms * occ * 8;  // about 8 waves of items
  return (int)std::max<int64_t>(1, std::min<int64_t>(nb, (pairs + want - 1) / want));
}

int pair_symm_sub(const inti_ctx* ctx, int tpt, int ch, int nitems) {
  // Parts of at least 32 sources (one FP32C group) until there are 16 CTAs
  // per SM: four waves of the four resident ones, so that the last, partly
  // filled one weighs little.  With whole blocks (78 CTAs at 3,072 nodes) a
  // Helmholtz SL took 64 us in the pair kernel; 27 us with eight parts.
  if (ch != 1) return 1;
  int sub = 1;
  while (sub < pair_symm_block(tpt) / kGroup && (int64_t)nitems * sub < (int64_t)16 * ctx->num_sms) sub *= 2;
  return sub;
}

int pair_launch(inti_ctx* ctx, const PairLaunch& L) {
  const int tile = pair_tile(L.precision);
  const int64_t npad = L.n_tiles * tile;
  const int tps = (int)((L.n_tiles + L.split - 1) / L.split);
  int launches = 0;
  dispatch(L.pde, L.kind, L.dim, [&](auto tag) {
    using T = decltype(tag);
    auto go = [&](auto rtag) {
      using R = decltype(rtag);
      constexpr int TILE = std::is_same<R, float>::value ? kTile32 : kTile64;
      const int pb = 256;
      {
        ProfScope ps(ctx, "pack");
        const unsigned gp = (unsigned)((npad + pb - 1) / pb);
        bool done = false;
        if constexpr (symm_x2<T, R>()) {
          if (L.symm) {
            launch_pdl(ctx->stream, gp, pb, 0, &pack_sources_x2<T::kind>, L.n, npad, L.scoords, L.snormals, L.sweights,
                       L.x, L.c1[0], L.c2[0], static_cast<float*>(L.packed));
            done = true;
          }
        }
        if (done) {
        } else if (L.symm && (T::kind == ADL || T::kind == HS)) {
          launch_pdl(ctx->stream, gp, pb, 0, &pack_sym_normal<T::pde, T::dim, R>, L.n, npad, L.scoords, L.snormals,
                     L.sweights, L.x, static_cast<R*>(L.packed));
        } else {
          launch_pdl(ctx->stream, gp, pb, 0, &pack_sources<T::pde, T::kind, T::dim, R>, L.n, npad, L.scoords, L.snormals,
                     L.sweights, L.x, make_double2(L.c1[0], L.c1[1]), make_double2(L.c2[0], L.c2[1]),
                     static_cast<R*>(L.packed));
        }
      }
      if constexpr (symm_kind<T>()) {
        if (L.symm) {
          SymArgs a;
          a.npad = npad;
          a.items = L.sym_launch ? L.sym_launch : L.sym_items;
          a.ids = L.sym_launch ? L.sym_launch_ids : nullptr;
          a.sub = L.sym_sub;
          a.packed = L.packed;
          a.ypart = L.partial;
          a.zpart = L.zpart;
          a.k = L.k;
          a.kT = L.k * kExpiTable / (2 * kPi);
          a.delta = 2 * kPi / kExpiTable;
          a.expi = std::is_same<R, float>::value ? (const void*)expi_table_f32(ctx) : (const void*)expi_table_f64(ctx);
          a.err = L.err_flag;
          ctx->flag_armed = true;
          size_t sm;
          void (*fn)(SymArgs);
          if constexpr (symm_x2<T, R>()) {
            sm = symm_x2_smem<T>();
            if (L.sym_sub > 1)
              fn = L.tpt == 2 ? &pair_symm_x2<T::kind, 2, true> : &pair_symm_x2<T::kind, 4, true>;
            else
              fn = L.tpt == 2 ? &pair_symm_x2<T::kind, 2, false> : &pair_symm_x2<T::kind, 4, false>;
          } else {
            sm = symm_smem<T, R>();
            if (L.sym_sub > 1)
              fn = L.tpt == 2 ? &pair_symm<T::pde, T::kind, T::dim, R, TILE, 2, true>
                              : &pair_symm<T::pde, T::kind, T::dim, R, TILE, 4, true>;
            else
              fn = L.tpt == 2 ? &pair_symm<T::pde, T::kind, T::dim, R, TILE, 2, false>
                              : &pair_symm<T::pde, T::kind, T::dim, R, TILE, 4, false>;
          }
          INTI_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
          a.zld = npad;
          a.zcol0 = 0;
          if (L.sym_npanels <= 1) {
            ProfScope pp(ctx, "pair");
            const int grid = (L.sym_launch ? L.sym_launch_items : L.sym_nitems) * L.sym_sub;
            if (grid > 0) launch_pdl(ctx->stream, (unsigned)grid, kBlock, sm, fn, a);
            launches = 2;
            return;
          }
          // panels one after another; after each, its partials are folded
          // into the running sums (fixed order: panels ascending)
          const int bt = pair_symm_block(L.tpt);
          const bool cplx = T::pde == HELMHOLTZ;
          INTI_CUDA(cudaMemsetAsync(L.sym_acc, 0, (size_t)L.m * (cplx ? 16 : 8), ctx->stream));
          a.zld = L.sym_zld;
          launches = 1;
          for (int p = 0; p < L.sym_npanels; ++p) {
            const SymPanel& P = L.sym_panels[p];
            int grid = P.nitems;
            a.items = L.sym_table + P.item_off;
            a.ids = nullptr;
            if (L.sym_launch) {
              grid = L.sym_launch_panels[2 * p + 1];
              a.items = L.sym_launch + 3 * L.sym_launch_panels[2 * p];
              a.ids = L.sym_launch_ids + L.sym_launch_panels[2 * p];
              INTI_CUDA(cudaMemsetAsync(L.partial, 0, L.sym_ypart_bytes, ctx->stream));
              INTI_CUDA(cudaMemsetAsync(L.zpart, 0, L.sym_zpart_bytes, ctx->stream));
            }
            a.zcol0 = (int64_t)P.col0 * bt;
            {
              ProfScope pp(ctx, "pair");
              if (grid > 0) fn<<<(unsigned)grid, kBlock, sm, ctx->stream>>>(a);
            }
            SymFold f;
            f.m = std::min<int64_t>(L.m, (int64_t)P.rows * bt);
            f.bt = bt;
            f.rowptr = L.sym_table + P.rowptr_off;
            f.rowitems = L.sym_table + P.rowitems_off;
            f.ypart = L.partial;
            f.zpart = L.zpart;
            f.zld = L.sym_zld;
            f.col0 = P.col0;
            f.ncols = P.ncols;
            f.acc = L.sym_acc;
            const unsigned gf = (unsigned)((f.m + kFoldNodes - 1) / kFoldNodes);
            const unsigned tf = kFoldNodes * kFoldSlices;
            ProfScope pf(ctx, "epilogue");
            if (std::is_same<R, float>::value) {
              if (cplx) pair_symm_fold_kernel<float4, true><<<gf, tf, 0, ctx->stream>>>(f);
              else pair_symm_fold_kernel<float2, false><<<gf, tf, 0, ctx->stream>>>(f);
            } else {
              if (cplx) pair_symm_fold_kernel<double2, true><<<gf, tf, 0, ctx->stream>>>(f);
              else pair_symm_fold_kernel<double, false><<<gf, tf, 0, ctx->stream>>>(f);
            }
            launches += 2;
          }
          return;
        }
      }
      if (L.symm) throw Error(INTI_E_UNSUPPORTED, "symmetric form of this kernel");
      FwdArgs a;
      a.m = L.m;
      a.n_tiles = L.n_tiles;
      a.tiles_per_split = tps;
      a.tcoords = L.tcoords;
      a.tnormals = L.tnormals;
      a.packed = L.packed;
      a.partial = L.partial;
      a.k = L.k;
      a.kT = L.k * kExpiTable / (2 * kPi);
      a.delta = 2 * kPi / kExpiTable;
      a.expi = std::is_same<R, float>::value ? (const void*)expi_table_f32(ctx) : (const void*)expi_table_f64(ctx);
      a.err = L.err_flag;
      ctx->flag_armed = true;
      size_t sm = fwd_smem<T, R>();
      auto fn = L.tpt == 2 ? &pair_forward<T::pde, T::kind, T::dim, R, TILE, 2>
                           : &pair_forward<T::pde, T::kind, T::dim, R, TILE, 4>;
      if constexpr (!std::is_same<R, float>::value) {
        if (L.tpt == 2 && L.split > L.n_tiles) {
          fn = &pair_forward<T::pde, T::kind, T::dim, R, kFineTile, 2>;
          sm = fwd_smem<T, R>(kFineTile);
          a.n_tiles = npad / kFineTile;
          a.tiles_per_split = (int)((a.n_tiles + L.split - 1) / L.split);
        }
      }
      INTI_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      const int64_t rows = fwd_rows(L.precision, L.tpt);
      dim3 grid((unsigned)((L.m + rows - 1) / rows), (unsigned)L.split);
      ProfScope pp(ctx, "pair");
      launch_pdl(ctx->stream, grid, kBlock, sm, fn, a);
      launches = 2;
    };
    if (L.precision == INTI_FP32C)
      go(float());
    else
      go(double());
  });
  INTI_CUDA(cudaGetLastError());
  ctx->launches += launches;
  return launches;
}

int pair_epilogue(inti_ctx* ctx, const PairLaunch& L, const inti_csr* corr, const double* x,
                  double* y, const double* alpha, const double* beta, const double* rowscale) {
  EpiArgs e;
  e.rowscale = rowscale;
  e.m = L.m;
  e.split = L.split;
  e.partial = L.partial;
  e.scale = pair_scale(L.pde, L.kind, L.dim);
  e.rowptr = corr ? corr->rowptr.as<int64_t>() : nullptr;
  e.col = corr ? corr->col.as<int32_t>() : nullptr;
  e.val = corr ? corr->val.as<double>() : nullptr;
  e.x = x;
  e.y = y;
  e.ar = alpha ? alpha[0] : 1.0;
  e.ai = alpha ? alpha[1] : 0.0;
  e.br = beta ? beta[0] : 0.0;
  e.bi = beta ? beta[1] : 0.0;
  e.beta_zero = (e.br == 0.0 && e.bi == 0.0);
  const EpiShape es = epi_shape(L.symm ? 1 : L.split);
  const bool cplx = L.pde == HELMHOLTZ;
  ProfScope pe(ctx, "epilogue");
  if (L.symm && L.sym_npanels > 1) {
    // the panels' running sums hold the whole pair product
    e.partial = L.sym_acc;
    e.split = 1;
    if (cplx)
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<double2, true>, e, es.nodes);
    else
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<double, false>, e, es.nodes);
    INTI_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return 1;
  }
  if (L.symm) {
    const unsigned gs = (unsigned)((L.m + kEpiNodes - 1) / kEpiNodes);
    const unsigned ts = kEpiNodes * kEpiSlices;
    SymEpi se;
    se.npad = L.n_tiles * pair_tile(L.precision);
    se.bt = pair_symm_block(L.tpt);
    se.lsub = 0;
    while ((1 << se.lsub) < L.sym_sub) ++se.lsub;
    se.rowptr = L.sym_rowptr;
    se.rowitems = L.sym_rowitems;
    se.zpart = L.zpart;
    if (L.precision == INTI_FP32C) {
      if (cplx)
        launch_pdl(ctx->stream, gs, ts, 0, &pair_symm_epilogue_kernel<float4, true>, e, se);
      else
        launch_pdl(ctx->stream, gs, ts, 0, &pair_symm_epilogue_kernel<float2, false>, e, se);
    } else {
      if (cplx)
        launch_pdl(ctx->stream, gs, ts, 0, &pair_symm_epilogue_kernel<double2, true>, e, se);
      else
        launch_pdl(ctx->stream, gs, ts, 0, &pair_symm_epilogue_kernel<double, false>, e, se);
    }
    INTI_CUDA(cudaGetLastError());
    ctx->launches += 1;
    return 1;
  }
  if (L.precision == INTI_FP32C) {
    if (cplx)
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<float4, true>, e, es.nodes);
    else
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<float2, false>, e, es.nodes);
  } else {
    if (cplx)
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<double2, true>, e, es.nodes);
    else
      launch_pdl(ctx->stream, es.blocks(L.m), es.threads(), es.smem(), &pair_epilogue_kernel<double, false>, e, es.nodes);
  }
  INTI_CUDA(cudaGetLastError());
  ctx->launches += 1;
  return 1;
}

bool pair_small_eligible(int precision, int64_t m, int64_t n) {
  // sources capped so that a lane's chain (n / (16 warps * 32 lanes)) stays short
  return precision == INTI_FP64 && (double)m * (double)n <= kSmallPairs && m > 0 && n > 0 && n <= 65536;
}

// log2 of the warps per target: until the CTAs fill the SMs, while a lane
// keeps at least four records.
static int pair_small_warps(int num_sms, int64_t m, int64_t n) {
  int lk = 0;
  while ((1 << lk) < kSmallWarps && (m << (lk + 1)) <= (int64_t)num_sms * kSmallWarps && n >= (int64_t)128 << (lk + 1)) ++lk;
  return lk;
}

int pair_small(inti_ctx* ctx, const PairLaunch& L, const inti_csr* corr, const double* x, double* y,
               const double* alpha, const double* beta, const double* rowscale) {
  EpiArgs e;
  e.rowscale = rowscale;
  e.m = L.m;
  e.split = 1;
  e.partial = nullptr;
  e.scale = pair_scale(L.pde, L.kind, L.dim);
  e.rowptr = corr ? corr->rowptr.as<int64_t>() : nullptr;
  e.col = corr ? corr->col.as<int32_t>() : nullptr;
  e.val = corr ? corr->val.as<double>() : nullptr;
  e.x = x;
  e.y = y;
  e.ar = alpha ? alpha[0] : 1.0;
  e.ai = alpha ? alpha[1] : 0.0;
  e.br = beta ? beta[0] : 0.0;
  e.bi = beta ? beta[1] : 0.0;
  e.beta_zero = (e.br == 0.0 && e.bi == 0.0);
  const SmallSources src{L.scoords, L.snormals, L.sweights, L.x, make_double2(L.c1[0], L.c1[1]),
                         make_double2(L.c2[0], L.c2[1])};
  const int lk = pair_small_warps(ctx->num_sms, L.m, L.n);
  const unsigned grid = (unsigned)((L.m + (kSmallWarps >> lk) - 1) / (kSmallWarps >> lk));
  const double2* expi = L.pde == HELMHOLTZ ? expi_table_f64(ctx) : nullptr;
  const double kT = L.k * kExpiTable / (2 * kPi), delta = 2 * kPi / kExpiTable;
  dispatch(L.pde, L.kind, L.dim, [&](auto tag) {
    using T = decltype(tag);
    ProfScope pp(ctx, "pair");
    constexpr int N = Rec<T::pde, T::kind, T::dim, double>::n;
    constexpr size_t sm = sizeof(double) * N * small_tile<N>();
    if (sm + (T::pde == HELMHOLTZ ? 17408 : 1024) > 48 * 1024)
      INTI_CUDA(cudaFuncSetAttribute(pair_small_kernel<T::pde, T::kind, T::dim>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    pair_small_kernel<T::pde, T::kind, T::dim><<<grid, 32 * kSmallWarps, sm, ctx->stream>>>(
        L.m, L.n, L.tcoords, L.tnormals, src, L.k, kT, delta, expi, lk, e);
  });
  INTI_CUDA(cudaGetLastError());
  ctx->launches += 1;
  return 1;
}

int pair_assemble(inti_ctx* ctx, const PairLaunch& L, double* out) {
  if (L.n > 65535 * 1024LL) throw Error(INTI_E_ARG, "assemble: too many source columns");
  if (L.kind == CF) throw Error(INTI_E_UNSUPPORTED, "assemble the DL and SL parts separately");
  dispatch(L.pde, L.kind, L.dim, [&](auto tag) {
    using T = decltype(tag);
    if constexpr (T::kind != CF) {
      dim3 grid((unsigned)((L.m + 255) / 256), (unsigned)L.n);
      assemble_kernel<T::pde, T::kind, T::dim><<<grid, 256, 0, ctx->stream>>>(
          L.m, L.n, L.tcoords, L.tnormals, L.scoords, L.snormals, L.sweights, L.k, out);
    }
  });
  INTI_CUDA(cudaGetLastError());
  ctx->launches += 1;
  return 1;
}

// Transpose: the roles of the two node sets swap; partial is split x n double2.
// ===========================================================================
// Allocation-free apply.
//
// Some callers cannot call cudaMalloc at the moment they need the operator:
// code running inside a framework whose caching allocator already owns nearly
// all device memory (so a fresh cudaMalloc fails or fragments it), and code
// that must not pay an allocation's latency or implicit synchronisation in a
// solver loop.  inti_apply_noalloc serves them:
// the caller passes every input and output as device pointers, and the
// scratch the pair product needs (packed source records and per-chunk partial
// sums) lives in one fixed array of kNoAllocScratchBytes declared below.  The
// module holds that array on every GPU that loads the library, until exit.
//
// The first call on a device resolves the array's device address with
// cudaGetSymbolAddress and uploads the e^{i m delta} tables into static
// device arrays; make that first call before any stream capture.  Every call
// on a device shares the array and leaves its contents behind: calls that
// overlap on the GPU (different streams, or different host threads) race
// on it.  Nothing in the array has to start at zero: the pack kernel writes
// every record (padding included) and the pair kernel writes every partial
// slot it owns; only the timeout flag is cleared at the start of each call.
// If a bounded wait of the pair kernel runs out, the epilogue writes NaN into
// every entry of y (with synchronize = 0 no status reports the timeout).
// ===========================================================================
constexpr size_t kNoAllocScratchBytes = 32u << 20;  // 32 MiB
constexpr size_t kNoAllocFlagBytes = 256;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
static __device__ __align__(16) double2 g_noalloc_expi64[kExpiTable];
static __device__ __align__(16) float2 g_noalloc_expi32[kExpiTable];

namespace {

struct NoAllocDevice {
  unsigned char* scratch = nullptr;
  const double2* expi64 = nullptr;
  const float2* expi32 = nullptr;
  int num_sms = 0;
};

std::mutex g_noalloc_mu;
NoAllocDevice g_noalloc_dev[64];

// Once per device, with that device current: resolve the static arrays'
// device addresses (the host-side names are not device addresses) and fill
// the phase tables.
const NoAllocDevice& noalloc_setup(int dev) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (dev < 0 || dev >= 64) throw Error(INTI_E_ARG, "device index out of range for the static scratch");
  NoAllocDevice& d = g_noalloc_dev[dev];
  if (d.scratch) return d;
  void* p = nullptr;
  INTI_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
  void* t64 = nullptr;
  INTI_CUDA(cudaGetSymbolAddress(&t64, g_noalloc_expi64));
  void* t32 = nullptr;
  INTI_CUDA(cudaGetSymbolAddress(&t32, g_noalloc_expi32));
  const auto c = expi_host(false), s = expi_host(true);
  std::vector<double2> h64(kExpiTable);
  std::vector<float2> h32(kExpiTable);
  for (int m = 0; m < kExpiTable; ++m) {
    h64[m] = make_double2((double)c[m], (double)s[m]);
    h32[m] = make_float2((float)c[m], (float)s[m]);
  }
  INTI_CUDA(cudaMemcpyToSymbol(g_noalloc_expi64, h64.data(), sizeof(double2) * kExpiTable));
  INTI_CUDA(cudaMemcpyToSymbol(g_noalloc_expi32, h32.data(), sizeof(float2) * kExpiTable));
  INTI_CUDA(cudaDeviceGetAttribute(&d.num_sms, cudaDevAttrMultiProcessorCount, dev));
  d.expi64 = static_cast<const double2*>(t64);
  d.expi32 = static_cast<const float2*>(t32);
  d.scratch = static_cast<unsigned char*>(p);
  return d;
}

}  // namespace

int apply_noalloc(int pde, int kind, int dim, double k, int precision, int64_t m, const double* tc,
                  const double* tn, int64_t n, const double* sc, const double* sn, const double* sw,
                  const int64_t* rowptr, const int32_t* col, const double* val, const double* x, double* y,
                  const double* alpha, const double* beta, cudaStream_t stream, int synchronize) {
  if (pde != INTI_LAPLACE && pde != INTI_HELMHOLTZ) throw Error(INTI_E_ARG, "unknown pde");
  if (kind < INTI_SL || kind > INTI_HS) throw Error(INTI_E_ARG, "unknown kernel");
  if (precision != INTI_FP64 && precision != INTI_FP32C) throw Error(INTI_E_ARG, "unknown precision");
  if (dim != 2 && dim != 3) throw Error(INTI_E_ARG, "dim must be 2 or 3");
  if (pde == INTI_HELMHOLTZ && dim != 3) throw Error(INTI_E_UNSUPPORTED, "Helmholtz is implemented in 3D only");
  if (m <= 0 || n <= 0) throw Error(INTI_E_ARG, "m and n must be positive");
  if (!tc || !sc || !sw || !x || !y) throw Error(INTI_E_ARG, "a required device pointer is NULL");
  if ((kind == DL || kind == HS) && !sn) throw Error(INTI_E_ARG, "this kernel needs source normals");
  if ((kind == ADL || kind == HS) && !tn) throw Error(INTI_E_ARG, "this kernel needs target normals");
  if ((rowptr || col || val) && !(rowptr && col && val))
    throw Error(INTI_E_ARG, "the correction needs rowptr, col and val together");
  int dev = 0;
  INTI_CUDA(cudaGetDevice(&dev));
  const NoAllocDevice& D = noalloc_setup(dev);
  const int64_t tile = pair_tile(precision);
  const int64_t n_tiles = (n + tile - 1) / tile;
  const size_t rec_bytes = (size_t)n_tiles * tile * pair_record_bytes(pde, kind, dim, precision);
  const size_t packed_bytes = (rec_bytes + 255) / 256 * 256;
  const size_t pbytes = (size_t)m * pair_partial_bytes(pde, precision);
  const size_t room = kNoAllocScratchBytes - kNoAllocFlagBytes;
  if (packed_bytes + pbytes > room)
    throw Error(INTI_E_ARG, "problem too large for the fixed " + std::to_string(kNoAllocScratchBytes >> 20) +
                                " MiB scratch of inti_apply_noalloc: needs " +
                                std::to_string(packed_bytes + pbytes) + " bytes (use inti_op_apply)");
  // source chunks: enough CTAs for ~2 waves, bounded by the scratch and the tiles
  const int64_t blocks = (m + fwd_rows(precision, kTPT) - 1) / fwd_rows(precision, kTPT);
  int64_t split = std::max<int64_t>(1, (2LL * D.num_sms * 4 + blocks - 1) / blocks);
  split = std::min<int64_t>({split, n_tiles, 64, (int64_t)((room - packed_bytes) / pbytes)});
  const int64_t tps = (n_tiles + split - 1) / split;
  split = (n_tiles + tps - 1) / tps;
  int* flag = reinterpret_cast<int*>(D.scratch);
  void* packed = D.scratch + kNoAllocFlagBytes;
  void* partial = D.scratch + kNoAllocFlagBytes + packed_bytes;
  INTI_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), stream));
  dispatch(pde, kind, dim, [&](auto tag) {
    using T = decltype(tag);
    auto go = [&](auto rtag) {
      using R = decltype(rtag);
      constexpr int TILE = std::is_same<R, float>::value ? kTile32 : kTile64;
      const int64_t npad = n_tiles * TILE;
      pack_sources<T::pde, T::kind, T::dim, R><<<(unsigned)((npad + 255) / 256), 256, 0, stream>>>(
          n, npad, sc, sn, sw, x, make_double2(1.0, 0.0), make_double2(0.0, 0.0), static_cast<R*>(packed));
      FwdArgs a;
      a.m = m;
      a.n_tiles = n_tiles;
      a.tiles_per_split = (int)tps;
      a.tcoords = tc;
      a.tnormals = tn;
      a.packed = packed;
      a.partial = partial;
      a.k = k;
      a.kT = k * kExpiTable / (2 * kPi);
      a.delta = 2 * kPi / kExpiTable;
      a.expi = std::is_same<R, float>::value ? (const void*)D.expi32 : (const void*)D.expi64;
      a.err = flag;
      const size_t sm = fwd_smem<T, R>();
      auto fn = &pair_forward<T::pde, T::kind, T::dim, R, TILE>;
      INTI_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      fn<<<dim3((unsigned)blocks, (unsigned)split), kBlock, sm, stream>>>(a);
    };
    if (precision == INTI_FP32C)
      go(float());
    else
      go(double());
  });
  EpiArgs e;
  e.m = m;
  e.split = (int)split;
  e.partial = partial;
  e.scale = pair_scale(pde, kind, dim);
  e.rowptr = rowptr;
  e.col = col;
  e.val = val;
  e.x = x;
  e.y = y;
  e.ar = alpha ? alpha[0] : 1.0;
  e.ai = alpha ? alpha[1] : 0.0;
  e.br = beta ? beta[0] : 0.0;
  e.bi = beta ? beta[1] : 0.0;
  e.beta_zero = (e.br == 0.0 && e.bi == 0.0);
  e.err = flag;
  const EpiShape es = epi_shape((int)split);
  const bool cplx = pde == HELMHOLTZ;
  if (precision == INTI_FP32C) {
    if (cplx)
      pair_epilogue_kernel<float4, true><<<es.blocks(m), es.threads(), es.smem(), stream>>>(e, es.nodes);
    else
      pair_epilogue_kernel<float2, false><<<es.blocks(m), es.threads(), es.smem(), stream>>>(e, es.nodes);
  } else {
    if (cplx)
      pair_epilogue_kernel<double2, true><<<es.blocks(m), es.threads(), es.smem(), stream>>>(e, es.nodes);
    else
      pair_epilogue_kernel<double, false><<<es.blocks(m), es.threads(), es.smem(), stream>>>(e, es.nodes);
  }
  INTI_CUDA(cudaGetLastError());
  if (synchronize) {
    INTI_CUDA(cudaStreamSynchronize(stream));
    int f = 0;
    INTI_CUDA(cudaMemcpy(&f, flag, sizeof(int), cudaMemcpyDeviceToHost));
    if (f) throw Error(INTI_E_TIMEOUT, "a device-side bounded wait ran out (code " + std::to_string(f) + ")");
  }
  return INTI_OK;
}

}  // namespace inti

extern "C" int inti_apply_noalloc(int pde, int kernel, int dim, double k, int precision, int64_t m,
                                  const double* tcoords, const double* tnormals, int64_t n,
                                  const double* scoords, const double* snormals, const double* sweights,
                                  const int64_t* rowptr, const int32_t* col, const double* val,
                                  const double* x, double* y, const double* alpha, const double* beta,
                                  void* stream, int synchronize) {
  try {
    return inti::apply_noalloc(pde, kernel, dim, k, precision, m, tcoords, tnormals, n, scoords, snormals,
                               sweights, rowptr, col, val, x, y, alpha, beta,
                               static_cast<cudaStream_t>(stream), synchronize);
  } catch (const inti::Error& e) {
    inti::noalloc_error_set(e.what());
    return e.code;
  } catch (const std::exception& e) {
    inti::noalloc_error_set(e.what());
    return INTI_E_ARG;
  }
}
