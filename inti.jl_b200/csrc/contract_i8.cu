// Multi-column pair contractions Y = K X with FP64 accuracy on the INT8
// tensor path (tcgen05 kind::i8): the product of an operator with many
// densities, the batched operators, and the Theta product of the
// density-interpolation correction.
//
// tcgen05 has no FP64 kind, and the FP64 MMA (mma.sync, fp64_mma.cuh) shares
// the 64-lane FP64 datapath with the kernel evaluation: 64 complex columns
// cost 256 FMA lanes a pair next to about 45 for the kernel value.  Here both
// factors are written as 64-bit fixed-point numbers in eight signed base-256
// digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59 (2012), with integer digits), the digit products run on the
// tensor cores with exact 32-bit integer sums, and the sums are put together
// in FP64 once per item.  What is left on the FP64 pipe is one kernel
// evaluation per pair and column group and four instructions per value that
// cut it into digits.
//
// Accuracy.  Row i of A = K is scaled by a power of two pa that takes a bound
// of |K_i.| to 2^61.9 .. 2^62.9, column c of B = diag(w) X by one (pb) for max
// |w x_c|; both are rounded to integers (error 1/2), the digit products with
// p + q <= 7 are kept (p, q = 0 the leading digits) and the mean of the others
// is added at the end (fx_mean).  Sums carry no rounding.  What is missing is at
// most 2^65.2 / (pa pb) per real product, whatever the product's own size: one
// scale serves a whole row and a whole column.  fx_guard therefore measures
// each result's sum of moduli T (with |r||n| in the place of |r.n|) against that
// unit, and the products in which
// an entry would come out worse than n 2^-52.8 T, the a priori bound of an FP64
// sum of n terms, are left to the FP64 kernels: unit vectors, narrow bumps,
// densities on one part of a surface, refined surfaces, targets close to a
// surface.  With smooth densities on uniform meshes the single and double
// layers and Theta lie 2^7 to 2^16 above the limit; the hypersingular kernel
// lies 2^2 to 2^7 above it with the 40 nearest sources of a target taken apart
// (fx_plan_near), and mostly below it without.  Far above, the result is closer to the exact product of the
// FP64 kernel values than an FP64 accumulation, which rounds n times at 2^-53
// of the running sum (64 columns, 13,872 nodes: 1.9e-15 from 64-bit values).  tests/test_gpu_contract_accuracy.py
// holds each entry to these bounds in extended precision.
//
// Work.  A persistent CTA per SM takes items (128 targets, a run of source
// stages) from a counter, the longest first.  A stage is 64 K elements: NA
// values per pair (1 real, 2 complex, 2 or 4 for the (S, D) pair of Theta)
// of 64/NA sources.  Warp roles as in mrhs_tc.cu:
//   * 16 generator warps: thread (row, quarter) evaluates 64/(4 NA) sources
//     for its row and writes eight 16-byte chunks (one per digit, 16 K
//     elements) of the A operand to shared memory: 128 rows x 16 B contiguous
//     per chunk, conflict-free;
//   * a copy warp: source records (FP64) and digit blocks of the densities
//     by the TMA bulk engine;
//   * an MMA warp: the digits of B lie one after another along N, so A's
//     digit p against B's digits 0..7-p is one wide product (N = (8-p) NC,
//     at most 256 per instruction) whose columns start at diagonal p of the
//     accumulators: eight diagonals of NC columns, all 512 tensor-memory
//     columns for NC = 64.  Reading each A digit once per 256 columns keeps
//     the operand traffic of shared memory below the MMA time.
// Only the integer, memory and conversion instructions of the generators
// overlap MMAs: on the B200 FP64 FMAs make no progress while INT8 MMAs are in
// flight (16 warps of independent FMAs next to an MMA loop: 1.5% of their rate
// alone, and the MMAs at 92% of theirs).  The MMAs of a stage therefore start
// once the values of the next stage are evaluated (aReady), and its packing
// and stores run beside them (two A buffers); starting them at once left the
// evaluation stalled and the packing alone (64 columns 1.92 -> 1.87 ms).  A
// stage costs about the sum: Theta with 18 complex columns 2,010 cycles of
// MMAs and stores (1,490 of operand reads), 1,990 of evaluation (1,353 of FP64
// issue) and 290 of hand-over.  The 32-bit sums
// hold 127 stages (8 * 255 * 128 * 8,128 < 2^31); then, or at the end of the
// item, the generators read the diagonals and add them up in FP64.
//
// More than 64 real columns go to pairs of CTAs that share the evaluation.
//
// Measured (B200, against the FP64 MMA kernels, device time): 64 complex
// columns of a Helmholtz DL at 13,872 nodes 5.63 -> 1.87 ms (2.48 without
// pairs); eight surfaces of 2,646 .. 21,600 nodes, combined field, 64 columns
// 26.9 -> 11.1 ms (15.7); the correction of a 43,200-node surface (18 complex
// columns) 33.6 -> 16.0 ms.
//
// e^{ikd} comes from a 128-entry table in eight copies, one per lane of a
// quarter-warp, so the gathers never conflict (a shared 1024-entry table
// costs about 12 wavefronts a warp, and shared memory is as busy here as the
// FP64 pipe), with one more term in the cosine.
//
// Every wait is bounded, as in mrhs_tc.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.h"
#include "contract_i8.h"
#include "device_common.cuh"
#include "internal.h"

namespace inti {

constexpr int FX_D = 8;                              // digits
constexpr int FX_K = 64;                             // K elements per stage
constexpr int FX_M = 128;                            // targets per item
constexpr int FX_NMAX = 64;                          // real columns per pass
constexpr int FX_GEN = 16;                           // generator warps
constexpr int FX_THREADS = 32 * (FX_GEN + 2);
constexpr int FX_FLUSH = 127;                        // stages a 32-bit sum holds
constexpr int FX_A_DIGIT = FX_M * FX_K;              // bytes of one digit of A
constexpr int FX_A_BYTES = FX_D * FX_A_DIGIT;        // 64 KB
constexpr int FX_B_BYTES = FX_D * FX_NMAX * FX_K;    // 32 KB
constexpr int FX_NS = 4;                             // source-record ring
constexpr int FX_ND = 4;                             // MMA completion ring
constexpr int FX_REC = 6;                            // doubles per source record
constexpr int FX_TAB = 128, FX_REP = 8;              // phase table, copies

template <int PDE, int KIND>
struct FxShape {
  static constexpr bool theta = KIND == FX_THETA || KIND == FX_THETA_D;
  static constexpr bool cplx = PDE == HELMHOLTZ;
  static constexpr int NA = (cplx ? 2 : 1) * (theta ? 2 : 1);
  static constexpr int J = FX_K / NA;        // sources per stage
  static constexpr int JT = J / 4;           // sources per generator thread and stage
  static constexpr bool tnormal = KIND == ADL || KIND == HS || KIND == FX_THETA_D;
  static constexpr bool near = KIND == HS || KIND == FX_THETA_D;  // nearest sources apart (fx_plan_near)
  static constexpr int S_BYTES = J * FX_REC * 8;
  static constexpr int OFF_B = 2 * FX_A_BYTES;
  static constexpr int OFF_T = OFF_B + 2 * FX_B_BYTES;
  static constexpr int OFF_S = OFF_T + (cplx ? FX_TAB * FX_REP * 16 : 0);
  static constexpr int SMEM = OFF_S + FX_NS * S_BYTES;
  static_assert(SMEM <= 230 * 1024, "shared memory");
};

static int fx_na(int pde, int kind) {
  return (pde == HELMHOLTZ ? 2 : 1) * (kind >= FX_THETA ? 2 : 1);
}

// Per-launch constants of the kernel values.
struct FxConst {
  double k, kT, c1r, c1i, c2r, c2i, kc1r, kc1i;
};

// e^{i d k}, kT = k FX_TAB / (2 pi): the table value of the nearest multiple
// of delta = 2 pi / FX_TAB times series of the rest (|r| = |f delta| <= H =
// pi/128): cos to r^6 (truncation below 4e-18), sin to r^5 with the r^7 term
// economised, x^7 ~ (112 x^5 - 56 x^3 + 7 x)/64 for x = r/H, which leaves
// H^7/5040/64 = 1.7e-17.
__device__ __forceinline__ void fx_expi(double d, double kT, const double2* __restrict__ tab, double& c, double& s) {
  constexpr double D = 2.0 * kPi / FX_TAB, D2 = D * D;
  constexpr double C2 = -D2 / 2, C4 = D2 * D2 / 24, C6 = -D2 * D2 * D2 / 720;
  constexpr double H2 = D2 / 4;
  constexpr double S1 = D * (1.0 - 7 * H2 * H2 * H2 / (64 * 5040.0)), S3 = D2 * D * (-1.0 / 6 + 56 * H2 * H2 / (64 * 5040.0)),
                   S5 = D2 * D2 * D * (1.0 / 120 - 112 * H2 / (64 * 5040.0));
  const double t = fma(d, kT, kRoundShift);
  const double f = fma(d, kT, -(t - kRoundShift));
  const double f2 = f * f;
  const double cp = fma(f2, fma(f2, fma(f2, C6, C4), C2), 1.0);
  const double sp = f * fma(f2, fma(f2, S5, S3), S1);
  const double2 e = tab[(__double2loint(t) & (FX_TAB - 1)) * FX_REP];
  c = fma(cp, e.x, -sp * e.y);
  s = fma(sp, e.x, cp * e.y);
}

// The squared distance that decides which pairs are taken apart: rounded the
// same way wherever it is asked for.
__device__ __forceinline__ double fx_dist2(double r0, double r1, double r2) {
  return __fma_rn(r2, r2, __fma_rn(r1, r1, __dmul_rn(r0, r0)));
}

// The NA values of one pair without the 1/(4 pi), times the row's scale p:
// (Re, Im) of the kernel, Theta: the S value(s), then the D value(s).  nx is
// the target normal times p.  rec = x y z nx ny nz of the
// source; e^{ikd}(1/d - ik)(r.n)/d^2 is formed as e^{ikd}(Q - ik P) with
// P = (r.n)/d^2, Q = P/d.  Pairs of a squared distance up to `cut` (bits; the
// self pair's, or that of the sources taken apart) are zero.
template <int PDE, int KIND>
__device__ __forceinline__ void fx_values(const double (&x)[3], const double (&nx)[3], double pr,
                                          const double* __restrict__ rec, const FxConst& c, const double2* __restrict__ tab,
                                          long long cut, double (&v)[FxShape<PDE, KIND>::NA]) {
  const double2 s01 = reinterpret_cast<const double2*>(rec)[0], s23 = reinterpret_cast<const double2*>(rec)[1];
  const double r0 = x[0] - s01.x, r1 = x[1] - s01.y, r2 = x[2] - s23.x;
  const double d2 = fx_dist2(r0, r1, r2);
  const double ri = __double_as_longlong(d2) > cut ? rsqrt_fast(d2) : 0.0;  // every value 0
  double rny = 0.0, rnx = 0.0, nn = 0.0;
  if (KIND != SL) {
    const double2 s45 = reinterpret_cast<const double2*>(rec)[2];
    if (KIND != ADL) rny = fma(r2, s45.y, fma(r1, s45.x, r0 * s23.y));
    if (FxShape<PDE, KIND>::tnormal) rnx = fma(r2, nx[2], fma(r1, nx[1], r0 * nx[0]));
    if (KIND == HS || KIND == FX_THETA_D) nn = fma(nx[2], s45.y, fma(nx[1], s45.x, nx[0] * s23.y));
  }
  const double id2 = ri * ri;
  if constexpr (PDE == LAPLACE) {
    const double ri3 = id2 * ri;
    if constexpr (KIND == SL)
      v[0] = pr * ri;
    else if constexpr (KIND == DL)
      v[0] = pr * rny * ri3;
    else if constexpr (KIND == ADL)
      v[0] = -rnx * ri3;
    else if constexpr (KIND == HS)
      v[0] = fma(-3.0 * rnx * rny, id2, nn) * ri3;
    else if constexpr (KIND == CF)
      v[0] = pr * fma(c.c2r, ri, c.c1r * (rny * ri3));
    else if constexpr (KIND == FX_THETA) {
      const double pri = pr * ri;
      v[0] = pri;
      v[1] = rny * (pri * id2);
    } else {
      v[0] = -rnx * ri3;
      v[1] = fma(-3.0 * rnx * rny, id2, nn) * ri3;
    }
  } else {
    const double d = d2 * ri;
    double cs, sn;
    fx_expi(d, c.kT, tab, cs, sn);
    auto times_e = [&](double wr, double wi, double& re, double& im) {
      re = fma(cs, wr, -sn * wi);
      im = fma(cs, wi, sn * wr);
    };
    auto layer = [&](double rn, double& re, double& im) {
      const double P = rn * id2;
      times_e(P * ri, -c.k * P, re, im);
    };
    auto hyper = [&](double& re, double& im) {
      // [(1/d - ik) p + (k^2 d^2 - 3 + 3ikd) s5], p = nn/d^2, s5 = rnx rny/d^5
      const double kd = c.k * d;
      const double p = nn * id2, s5 = (rnx * rny) * (id2 * id2 * ri);
      times_e(fma(ri, p, fma(kd, kd, -3.0) * s5), fma(-c.k, p, 3.0 * kd * s5), re, im);
    };
    if constexpr (KIND == SL) {
      const double pri = pr * ri;
      v[0] = pri * cs;
      v[1] = pri * sn;
    } else if constexpr (KIND == DL) {
      layer(pr * rny, v[0], v[1]);
    } else if constexpr (KIND == ADL) {
      layer(-rnx, v[0], v[1]);
    } else if constexpr (KIND == HS) {
      hyper(v[0], v[1]);
    } else if constexpr (KIND == CF) {
      const double P = rny * id2, Q = P * ri;
      const double cp = pr * cs, sp = pr * sn;
      const double wr = fma(c.c2r, ri, fma(c.c1r, Q, c.kc1i * P)), wi = fma(c.c2i, ri, fma(c.c1i, Q, -c.kc1r * P));
      v[0] = fma(cp, wr, -sp * wi);
      v[1] = fma(cp, wi, sp * wr);
    } else if constexpr (KIND == FX_THETA) {
      // D = (r.n)/d^2 (1 - ikd) S
      const double pri = pr * ri, kd = c.k * d, q = rny * id2;
      v[0] = pri * cs;
      v[1] = pri * sn;
      v[2] = q * fma(kd, v[1], v[0]);
      v[3] = q * fma(-kd, v[0], v[1]);
    } else {
      layer(-rnx, v[0], v[1]);
      hyper(v[2], v[3]);
    }
  }
}

// Power of two p with |v| p < 2^63 (1 - 2^-5) for |v| <= cur: eight balanced
// digits reach 0.498 * 2^64.  0 for cur = 0.
__device__ __forceinline__ double fx_scale(double cur) {
  if (!(cur > 0.0)) return 0.0;
  const long long b = __double_as_longlong(cur);
  const int e = (int)(b >> 52) - 1023;
  const bool high = (b & 0xFFFFFFFFFFFFFLL) > 0xE666666666666LL;  // mantissa above 1.9
  return __longlong_as_double((long long)(1023 + (high ? 61 : 62) - e) << 52);
}
// 0, or a magnitude whose scale and products of scales stay normal numbers.
__device__ __forceinline__ bool fx_fits(double cur) { return cur == 0.0 || (cur > 1e-120 && cur < 1e120); }

// Digits of A: the bytes of v rounded to a 64-bit integer, the leading one
// signed, the others unsigned (the MMA takes the signedness of A per
// instruction, so nothing has to be balanced: that took 2% of a product and
// 4% of Theta, and the mean of the dropped products is added in the end,
// fx_mean).  The conversion runs on the otherwise idle conversion unit;
// cutting v with rounding additions took four FP64 instructions.
__device__ __forceinline__ uint2 fx_bytes(double v) {
  const long long w = __double2ll_rn(v);
  return make_uint2((uint32_t)w, (uint32_t)(w >> 32));
}

// Digits of B are balanced (-128 .. 127): the bytes of the integer plus 0x80
// in every byte, each minus 128.
__device__ __forceinline__ uint2 fx_digits(double v) {
  const unsigned long long w = ((unsigned long long)__double2ll_rn(v) + 0x8080808080808080ULL) ^ 0x8080808080808080ULL;
  return make_uint2((uint32_t)w, (uint32_t)(w >> 32));
}

// Digits of four values as one word per digit (value e in byte e), leading
// digit first.
__device__ __forceinline__ void fx_pack4(const uint2 (&a)[4], uint32_t (&w)[FX_D]) {
  auto four = [](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t& b0, uint32_t& b1, uint32_t& b2,
                 uint32_t& b3) {
    const uint32_t l0 = __byte_perm(a0, a1, 0x5140), l1 = __byte_perm(a2, a3, 0x5140);
    const uint32_t h0 = __byte_perm(a0, a1, 0x7362), h1 = __byte_perm(a2, a3, 0x7362);
    b0 = __byte_perm(l0, l1, 0x5410);
    b1 = __byte_perm(l0, l1, 0x7632);
    b2 = __byte_perm(h0, h1, 0x5410);
    b3 = __byte_perm(h0, h1, 0x7632);
  };
  four(a[0].x, a[1].x, a[2].x, a[3].x, w[7], w[6], w[5], w[4]);
  four(a[0].y, a[1].y, a[2].y, a[3].y, w[3], w[2], w[1], w[0]);
}

// ---------------------------------------------------------------------------
// tensor-core primitives
// ---------------------------------------------------------------------------
// K-major, no swizzle: 8-row x 16-byte core matrices, `lbo` bytes between
// K chunks, 128 bytes between 8-row groups.
__device__ __forceinline__ uint64_t fx_desc(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)((lbo >> 4) & 0x3FFF) << 16 | (uint64_t)(128 >> 4) << 32 |
         (uint64_t)1 << 46;
}

// S32 accumulate, 8-bit A (signed or not) and signed B, both K-major, M = 128
__host__ __device__ constexpr uint32_t fx_idesc(int n, bool a_signed) {
  return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(FX_M >> 4) << 24);
}

__device__ __forceinline__ void fx_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ bool fx_elect() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.b32 %0, 1, 0, P;\n\t}" : "=r"(e));
  return e != 0;
}

__device__ __forceinline__ void fx_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void fx_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fx_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void fx_ld4(uint32_t taddr, int32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr));
}
__device__ __forceinline__ void fx_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// --- pairs of CTAs ---------------------------------------------------------
__device__ __forceinline__ uint32_t fx_peer(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void fx_st_peer(uint32_t a, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// Bulk copy from this CTA's shared memory to the peer's, completing on a
// barrier of the peer (mapped addresses; 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void fx_copy_peer(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "r"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fx_commit_both(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void fx_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// mbar_wait_bounded for a barrier that the peer arrives at, too.
template <int CL>
__device__ __forceinline__ bool fx_wait(uint64_t* bar, uint32_t parity) {
  if (CL == 1) return mbar_wait_bounded(bar, parity);
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

struct FxArgs {
  const FxRows* rows;
  const FxItem* items;
  int nitems;
  int nc;                   // real columns of this pass (fx_width)
  const double* tcoords;
  const double* tnormals;
  const double* rowscale;   // per target
  const double* cut2;       // per target, for kernels with sources apart
  const double* records;    // source records, J per stage
  const unsigned char* bdig;  // digit blocks, nc * 512 bytes per stage, one plane per CTA of a pair
  int nstages;                // stages of a plane
  const double2* tab;       // FX_TAB phase table
  double* partial;          // [CTA of the pair][slot][column][128]
  int nslots;
  FxConst c;
  int* counter;
  const int* flag;
  int* err;
};

// The MMAs of one stage: A digit p against the digits 0 .. 7-p of B, in equal
// parts of at most 256 columns, for each K slab of 32 elements.  Digit 0 covers every
// accumulator column, so its first slab may overwrite them (accumulate 0).
// For odd NC/8 a product of an odd number of digits is rounded up by eight
// columns: they read the digit after and add to the columns past the last
// diagonal, which nothing reads.
// Unrolled, so that every offset is an immediate: the issuing lane competes
// with the generators for its issue slots, and a loop that reads them from
// shared memory took about 330 cycles per MMA, three times the MMA's own.
template <int NC>
__device__ __forceinline__ void fx_issue(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t accumulate) {
#pragma unroll
  for (int slab = 0; slab < 2; ++slab) {
#pragma unroll
    for (int p = 0; p < FX_D; ++p) {
      const int total = ((FX_D - p) * NC + 15) / 16 * 16, parts = (total + 255) / 256;
      const int w = (total / parts + 15) / 16 * 16;
      static_assert(NC % 8 == 0 && 8 * NC + (NC % 16 ? 8 : 0) <= 512, "tensor memory");
#pragma unroll
      for (int part = 0; part < parts; ++part) {
        const int n0 = part * w, n = min(w, total - n0);
        fx_mma(tmem + p * NC + n0, ad + ((p * FX_A_DIGIT + slab * 2 * FX_M * 16) >> 4),
               bd + ((slab * 2 * NC * FX_D * 16 + n0 * 16) >> 4), fx_idesc(n, p == 0),
               slab == 0 && p == 0 ? accumulate : 1u);
      }
    }
  }
}

// Sum of the diagonals of one accumulator element in units of 256^7.
__device__ __forceinline__ double fx_sum(const int32_t (&d)[FX_D][4], int e) {
  const long long hi = ((long long)d[0][e] << 24) + ((long long)d[1][e] << 16) + ((long long)d[2][e] << 8) + d[3][e];
  const long long lo = ((long long)d[4][e] << 24) + ((long long)d[5][e] << 16) + ((long long)d[6][e] << 8) + d[7][e];
  return fma((double)hi, 4294967296.0, (double)lo);
}

// CL = 2: a cluster of two CTAs works on the same items, each for its own
// columns (up to 64 each).  Each evaluates half of a stage's pairs (two of the
// four chunks) and the copy warp sends the digits to the other's A buffer (a
// 4 KB bulk copy per digit), so that a kernel value is made once for 128
// columns.  The MMAs of both must be done before either buffer is written
// again: mmaDone counts two commits.  (Stores of the generators straight into
// the peer's shared memory were twice as slow as evaluating everything twice.)
template <int PDE, int KIND, int CL>
__global__ void __launch_bounds__(FX_THREADS, 1) fx_contract_kernel(FxArgs a) {
  pdl_wait();
  using SH = FxShape<PDE, KIND>;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ __align__(8) uint64_t fullS[FX_NS], fullB[2], aReady[2], aFull[2], aPeer[2], mmaDone[FX_ND], drainBar;
  __shared__ uint32_t tmem_base_sh;
  __shared__ int item_sh, fail_sh;
  if (*a.flag) return;  // densities or kernel values out of range: the FP64 kernels run
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nc = a.nc;
  const uint32_t rank = CL == 2 ? blockIdx.x & 1 : 0;  // clusters are consecutive blocks
  const unsigned char* bdig = a.bdig + (size_t)rank * a.nstages * nc * (FX_D * FX_K);
  double* partial = a.partial + (size_t)rank * a.nslots * nc * FX_M;
  const uint32_t bstage = (uint32_t)nc * (FX_D * FX_K), blbo = (uint32_t)nc * (FX_D * 16);
  if (tid == 0) {
    for (int q = 0; q < FX_NS; ++q) mbar_init(&fullS[q], 1);
    for (int q = 0; q < FX_ND; ++q) mbar_init(&mmaDone[q], CL);
    for (int q = 0; q < 2; ++q) {
      mbar_init(&fullB[q], 1);
      mbar_init(&aReady[q], FX_GEN);
      mbar_init(&aFull[q], FX_GEN);
      mbar_init(&aPeer[q], 1);
    }
    fail_sh = 0;
    mbar_init(&drainBar, 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (SH::cplx) {
    double2* tab = reinterpret_cast<double2*>(sm + SH::OFF_T);
    for (int q = tid; q < FX_TAB * FX_REP; q += FX_THREADS) tab[q] = a.tab[q / FX_REP];
  }
  fx_fence_before();
  __syncthreads();
  fx_fence_after();
  if (CL == 2) fx_cluster_sync();  // the peer's barriers are there
  const uint32_t tmem = tmem_base_sh, sbase = smem_u32(sm);

  uint32_t g = 0;           // stages done by this CTA (same in every thread)
  uint32_t nS = 0, nB = 0;  // copy warp: copies issued
  uint32_t nC = 0;          // MMA warp: groups committed
  uint32_t nA = 0;          // copy warp: stages sent to the peer (and awaited from it)
  bool ok = true;

  for (;;) {
    if (tid == 0 && rank == 0) {
      const int next = atomicAdd(a.counter, 1);
      item_sh = next;
      if (CL == 2) fx_st_peer(fx_peer(smem_u32(&item_sh), 1), (uint32_t)next);
    }
    if (CL == 2)
      fx_cluster_sync();
    else
      __syncthreads();
    const int it = item_sh;
    if (it >= a.nitems) break;
    const FxItem item = a.items[it];
    const FxRows rb = a.rows[item.rows];
    for (int done = 0; done < item.nstages; done += FX_FLUSH) {
      const uint32_t T = (uint32_t)min(FX_FLUSH, item.nstages - done);
      const int64_t st0 = (int64_t)rb.stage0 + item.stage + done;
      if (warp == 0) {
        for (uint32_t t = 0; t < T; ++t) {
          const uint32_t gg = g + t, bb = gg & 1;
          ok = mbar_wait_bounded(&aFull[bb], (gg >> 1) & 1) && mbar_wait_bounded(&fullB[bb], (gg >> 1) & 1) &&
               (CL == 1 || fx_wait<CL>(&aPeer[bb], (gg >> 1) & 1)) &&
               (t + 1 == T || mbar_wait_bounded(&aReady[bb ^ 1], ((gg + 1) >> 1) & 1));
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          fx_fence_after();
          if (fx_elect()) {
            const uint64_t ad = fx_desc(sbase + bb * FX_A_BYTES, FX_M * 16);
            const uint64_t bd = fx_desc(sbase + SH::OFF_B + bb * FX_B_BYTES, blbo);
            const uint32_t acc = t > 0 ? 1u : 0u;
            switch (nc) {
              case 16: fx_issue<16>(tmem, ad, bd, acc); break;
              case 24: fx_issue<24>(tmem, ad, bd, acc); break;
              case 32: fx_issue<32>(tmem, ad, bd, acc); break;
              case 40: fx_issue<40>(tmem, ad, bd, acc); break;
              case 48: fx_issue<48>(tmem, ad, bd, acc); break;
              case 56: fx_issue<56>(tmem, ad, bd, acc); break;
              default: fx_issue<64>(tmem, ad, bd, acc); break;
            }
            if (CL == 2)
              fx_commit_both(&mmaDone[gg % FX_ND]);
            else
              fx_commit(&mmaDone[gg % FX_ND]);
          }
          __syncwarp();
          ++nC;
        }
      } else if (warp == 1) {
        auto copyS = [&](uint32_t t) {
          const uint32_t b = (g + t) % FX_NS;
          if (fx_elect()) {
            mbar_arrive_expect_tx(&fullS[b], SH::S_BYTES);
            bulk_copy_g2s(sm + SH::OFF_S + b * SH::S_BYTES, a.records + (st0 + t) * (SH::J * FX_REC), SH::S_BYTES,
                          &fullS[b]);
          }
          __syncwarp();
          ++nS;
        };
        auto copyB = [&](uint32_t t) {
          const uint32_t b = (g + t) & 1;
          if (fx_elect()) {
            mbar_arrive_expect_tx(&fullB[b], bstage);
            bulk_copy_g2s(sm + SH::OFF_B + b * FX_B_BYTES, bdig + (size_t)(st0 + t) * bstage, bstage, &fullB[b]);
          }
          __syncwarp();
          ++nB;
        };
        // the buffers of the run before are free: its MMAs were waited for
        for (uint32_t t = 0; t < FX_NS - 1 && t < T; ++t) copyS(t);
        copyB(0);
        for (uint32_t t = 0; t + 1 < T || (CL == 2 && t < T); ++t) {
          if (CL == 2) {  // this CTA's chunks of the stage to the peer
            const uint32_t bb = (g + t) & 1;
            ok = mbar_wait_bounded(&aFull[bb], ((g + t) >> 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) {
              ok = false;
              break;
            }
            if (fx_elect()) {
              constexpr uint32_t kHalf = FX_A_DIGIT / 2;
              mbar_arrive_expect_tx(&aPeer[bb], FX_D * kHalf);
              const uint32_t src = sbase + bb * FX_A_BYTES + rank * kHalf;
              const uint32_t dst = fx_peer(src, rank ^ 1), bar = fx_peer(smem_u32(&aPeer[bb]), rank ^ 1);
#pragma unroll
              for (int p = 0; p < FX_D; ++p) fx_copy_peer(dst + p * FX_A_DIGIT, src + p * FX_A_DIGIT, kHalf, bar);
            }
            __syncwarp();
            ++nA;
            if (t + 1 >= T) break;
          }
          // MMA group gg-1 read the B buffer of stage gg+1 and, through its A
          // tile, the source records of stage gg-1
          const uint32_t gg = g + t;
          if (t > 0) ok = fx_wait<CL>(&mmaDone[(gg - 1) % FX_ND], ((gg - 1) / FX_ND) & 1);
          if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
          }
          copyB(t + 1);
          if (t + FX_NS - 1 < T) copyS(t + FX_NS - 1);
        }
      } else {
        const int gw = warp - 2, quarter = gw >> 2;
        const int r = 32 * (warp & 3) + lane;  // target row = tensor-memory lane
        const int64_t row = rb.row0 + min(r, rb.nrows - 1);
        double x[3], nx[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int c = 0; c < 3; ++c) x[c] = a.tcoords[3 * row + c];
        if (SH::tnormal) {
#pragma unroll
          for (int c = 0; c < 3; ++c) nx[c] = a.tnormals[3 * row + c] * a.rowscale[row];
        }
        const double scale = a.rowscale[row];
        const long long cut = __double_as_longlong(SH::near ? a.cut2[row] : kSamePointTol2);
        const double2* tab = reinterpret_cast<const double2*>(sm + SH::OFF_T) + (lane & (FX_REP - 1));
        for (uint32_t t = 0; t < T; ++t) {
          const uint32_t gg = g + t, sb = gg % FX_NS;
          bool w = mbar_wait_bounded(&fullS[sb], (gg / FX_NS) & 1);
          if (!__all_sync(0xffffffffu, w)) {
            ok = false;
            break;
          }
          // a pair: chunks 2 rank, 2 rank + 1, half of a chunk's groups per thread
          const int chunk = CL == 2 ? (int)rank * 2 + (quarter >> 1) : quarter;
          const double* S = reinterpret_cast<const double*>(sm + SH::OFF_S + sb * SH::S_BYTES) +
                            chunk * SH::JT * FX_REC;
          unsigned char* A = sm + (gg & 1) * FX_A_BYTES + chunk * (FX_M * 16) + r * 16;
          // Groups of four sources, NA words each.  The octets of a warp take
          // them in rotated order, so that their stores of NA words at a
          // stride of 16 bytes fall on distinct banks.
          constexpr int G = SH::JT / 4, GQ = G / CL;  // of a chunk; of this thread
          static_assert(GQ >= 1, "a group per thread");
          const int g0 = (CL == 2 ? (quarter & 1) * GQ : 0) + (lane >> 3);
          uint2 dg[GQ][SH::NA][4];
#pragma unroll
          for (int q = 0; q < GQ; ++q) {
            const double* Sg = S + ((q + g0) & (G - 1)) * (4 * FX_REC);
            double v[4][SH::NA];
#pragma unroll
            for (int e = 0; e < 4; ++e) fx_values<PDE, KIND>(x, nx, scale, Sg + e * FX_REC, a.c, tab, cut, v[e]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
              for (int n = 0; n < SH::NA; ++n) dg[q][n][e] = fx_bytes(v[e][n]);
          }
          // FP64 work of the stage done: the MMAs of the one before may run,
          // beside the packing of this one
#pragma unroll
          for (int q = 0; q < GQ; ++q)
#pragma unroll
            for (int n = 0; n < SH::NA; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e) asm volatile("" : "+r"(dg[q][n][e].x), "+r"(dg[q][n][e].y));
          __syncwarp();
          if (lane == 0) mbar_arrive(&aReady[gg & 1]);
          // A buffer gg & 1 was last read by MMA group gg-2
          if (t >= 2) w = fx_wait<CL>(&mmaDone[(gg - 2) % FX_ND], ((gg - 2) / FX_ND) & 1);
          if (!__all_sync(0xffffffffu, w)) {
            ok = false;
            break;
          }
#pragma unroll
          for (int q = 0; q < GQ; ++q) {
            uint32_t wd[SH::NA][FX_D];
#pragma unroll
            for (int n = 0; n < SH::NA; ++n) fx_pack4(dg[q][n], wd[n]);
            unsigned char* Ag = A + ((q + g0) & (G - 1)) * (4 * SH::NA);
#pragma unroll
            for (int p = 0; p < FX_D; ++p) {
              if constexpr (SH::NA == 1)
                *reinterpret_cast<uint32_t*>(Ag + p * FX_A_DIGIT) = wd[0][p];
              else if constexpr (SH::NA == 2)
                *reinterpret_cast<uint2*>(Ag + p * FX_A_DIGIT) = make_uint2(wd[0][p], wd[1][p]);
              else
                *reinterpret_cast<uint4*>(Ag + p * FX_A_DIGIT) = make_uint4(wd[0][p], wd[1][p], wd[2][p], wd[3][p]);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&aFull[gg & 1]);
        }
        if (ok) {
          const uint32_t gl = g + T - 1;
          ok = __all_sync(0xffffffffu, fx_wait<CL>(&mmaDone[gl % FX_ND], (gl / FX_ND) & 1));
        }
        if (ok) {
          fx_fence_after();
          const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
          double* out = partial + (size_t)item.slot * nc * FX_M + r;
          for (int c = 4 * quarter; c < nc; c += FX_GEN) {
            int32_t d[FX_D][4];
#pragma unroll
            for (int s = 0; s < FX_D; ++s) fx_ld4(lane_addr + s * nc + c, d[s]);
            fx_wait_ld();
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              double v = fx_sum(d, e);
              double* o = out + (size_t)(c + e) * FX_M;
              if (done > 0) v += *o;  // the runs of an item add up in the same thread
              *o = v;
            }
          }
        }
      }
      g += T;
      fx_fence_before();
      // accumulators read (or the run abandoned, by both CTAs) before the next run's MMAs
      if (CL == 2) {
        if (!ok) {
          fail_sh = 1;
          fx_st_peer(fx_peer(smem_u32(&fail_sh), rank ^ 1), 1u);
        }
        fx_cluster_sync();
        if (*(volatile int*)&fail_sh) goto fail;
      } else if (__syncthreads_or(!ok)) {
        goto fail;
      }
      fx_fence_after();
    }
  }
  goto done;
fail:
  if (tid == 0) atomicExch(a.err, kErrWaitTimeout);
  // Everything this CTA put in flight must land before it leaves (each copy
  // alone on its barrier; one more commit tracks every MMA issued).
  if (warp == 1 && lane == 0) {
    for (uint32_t q = nS > FX_NS ? nS - FX_NS : 0; q < nS; ++q) mbar_wait_bounded(&fullS[q % FX_NS], (q / FX_NS) & 1);
    for (uint32_t q = nB > 2 ? nB - 2 : 0; q < nB; ++q) mbar_wait_bounded(&fullB[q & 1], (q >> 1) & 1);
    for (uint32_t q = nA > 2 ? nA - 2 : 0; q < nA; ++q) mbar_wait_bounded(&aPeer[q & 1], (q >> 1) & 1);
  }
  if (warp == 0) {
    if (nC > 0 && fx_elect()) {
      fx_commit(&drainBar);
      mbar_wait_bounded(&drainBar, 0);
    }
    __syncwarp();
  }
  __syncthreads();
done:
  fx_fence_before();
  __syncthreads();
  if (CL == 2) fx_cluster_sync();  // neither leaves while the other may still reach its shared memory
  if (warp == 0) {
    fx_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
  }
}

// ---------------------------------------------------------------------------
// plan kernels
// ---------------------------------------------------------------------------
// Centre and radius of each stage's sources (double4), their least normal and
// their records; the largest normal of all sources (bits in meta[0]).
__global__ void fx_plan_sources(int nstages, int J, const FxStage* __restrict__ stages,
                                const double* __restrict__ coords, const double* __restrict__ normals,
                                double* __restrict__ records, double4* __restrict__ tiles,
                                double* __restrict__ least_normal, unsigned long long* __restrict__ meta) {
  const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (s >= nstages) return;
  const FxStage st = stages[s];
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY}, n2 = 0.0,
         least = INFINITY;
  for (int j = lane; j < J; j += 32) {
    double v[FX_REC] = {0, 0, 0, 0, 0, 0};
    if (j < st.count) {
      const int64_t i = st.src0 + j;
      for (int c = 0; c < 3; ++c) {
        v[c] = coords[3 * i + c];
        lo[c] = fmin(lo[c], v[c]);
        hi[c] = fmax(hi[c], v[c]);
        if (normals) v[3 + c] = normals[3 * i + c];
      }
      const double q2 = v[3] * v[3] + v[4] * v[4] + v[5] * v[5];
      n2 = fmax(n2, q2);
      least = fmin(least, q2);
    }
    for (int c = 0; c < FX_REC; ++c) records[((int64_t)s * J + j) * FX_REC + c] = v[c];
  }
  for (int o = 16; o > 0; o >>= 1) {
    for (int c = 0; c < 3; ++c) {
      lo[c] = fmin(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = fmax(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
    n2 = fmax(n2, __shfl_xor_sync(0xffffffffu, n2, o));
    least = fmin(least, __shfl_xor_sync(0xffffffffu, least, o));
  }
  if (lane == 0) {
    least_normal[s] = sqrt(least);
    const double a = hi[0] - lo[0], b = hi[1] - lo[1], c = hi[2] - lo[2];
    tiles[s] = make_double4((lo[0] + hi[0]) / 2, (lo[1] + hi[1]) / 2, (lo[2] + hi[2]) / 2,
                            0.5 * sqrt(a * a + b * b + c * c) * (1 + 1e-12));
    atomicMax(meta, (unsigned long long)__double_as_longlong(sqrt(n2)));
  }
}

// The larger value; a NaN (of a coefficient that is not finite) stays.
__device__ __forceinline__ double fx_max(double a, double b) { return b > a || b != b ? b : a; }

// Bound of |K(x, y)| over the NA values from the modulus of the kernel (no
// phase), with the distance d, id = 1/d, |r.n_x|, |r.n_y| and |n_x.n_y| given.
template <int PDE, int KIND>
__device__ __forceinline__ double fx_modulus(double d, double id, double rnx, double rny, double nn,
                                             const FxConst& c) {
  const double id2 = id * id;
  const double k = PDE == HELMHOLTZ ? fabs(c.k) : 0.0;
  const double f = (id + k) * id2;  // |e^{ikd}(1/d - ik)|/d^2 at most
  const double h = f * nn + ((k * d) * (k * d) + 3.0 + 3.0 * k * d) * rnx * rny * (id2 * id2 * id);
  if (KIND == SL) return id;
  if (KIND == DL) return f * rny;
  if (KIND == ADL) return f * rnx;
  if (KIND == HS) return h;
  if (KIND == CF) return (fabs(c.c1r) + fabs(c.c1i)) * f * rny + (fabs(c.c2r) + fabs(c.c2i)) * id;
  if (KIND == FX_THETA) return fx_max(id, f * rny);
  return fx_max(f * rnx, h);
}

// The hypersingular kernel's nearest values, about 1/h^3, set a row's scale
// while the entry may rest on values far smaller.  The sources about a target
// are therefore taken apart: cut2 is a squared distance about the target, its
// entries (pairs closer than that, up to kNear) are kept with their kernel
// values, multiplied in FP64 (fx_near_add), and zero in the contraction.  The
// rest of the row is then at most 1/(3.5h)^3: on spheres of 1,728 .. 13,872 and
// ellipsoids of 1,944 .. 15,606 nodes the least sum of moduli of an entry rises
// from 2^-13 .. 2^-5 of the two scales to 2^-5 .. 2^-1.  64 complex columns of
// 13,872 nodes: 5.90 ms on the FP64 MMA path, 2.12 ms here; the derivative
// correction of 43,200 nodes 34.0 and 17.4 ms.  Plan (once per operator, 0.1 ms
// there) and entries (40 values per target) pay from the sizes of fx_pays.
constexpr int kNear = 48;       // entries per target at most
constexpr double kNearFill = 40.0 / kPi;  // cut2 / the nearest source's weight: some 40 of a surface's sources

struct FxNear {
  int32_t* count;    // per target
  int32_t* idx;      // entry e of target r at e * estep + r * rstep
  double* val;       // there times NV: (Re, Im) of the kernel, FX_THETA_D: of both
  int64_t estep, rstep;
};

// Kernel values of one entry times the source's weight, without the 1/(4 pi):
// e^{ikd} [(1/d - ik) p + (k^2 d^2 - 3 + 3ikd) q], p = nn/d^2, q = rnx rny/d^5.
template <int PDE, int KIND>
__device__ __forceinline__ void fx_near_values(const double (&x)[3], const double (&nx)[3], const double* __restrict__ y,
                                               const double* __restrict__ ny, double w, double k, double* v) {
  constexpr bool TH = FxShape<PDE, KIND>::theta;
  constexpr int NV = FxShape<PDE, KIND>::NA;
  double d2 = 0.0, rnx = 0.0, rny = 0.0, nn = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double r = x[c] - y[c], n = ny[c];
    d2 = fma(r, r, d2);
    rnx = fma(r, nx[c], rnx);
    rny = fma(r, n, rny);
    nn = fma(nx[c], n, nn);
  }
  const double d = sqrt(d2), id1 = 1.0 / d, id2 = 1.0 / d2;
  const double p = w * (nn * id2), q = w * (rnx * rny * (id2 * id2 * id1)), a = -w * (rnx * id2);
  if constexpr (PDE == LAPLACE) {
    if (TH) v[0] = a * id1;
    v[NV - 1] = fma(-3.0, q, p * id1);
  } else {
    const double kd = k * d;
    double s, c;
    sincos(kd, &s, &c);
    auto put = [&](double wr, double wi, double* o) {
      o[0] = fma(c, wr, -s * wi);
      o[1] = fma(c, wi, s * wr);
    };
    if (TH) put(a * id1, -k * a, v);
    put(fma(id1, p, fma(kd, kd, -3.0) * q), fma(-k, p, 3.0 * kd * q), v + NV - 2);
  }
}

// One warp per target.
template <int PDE, int KIND>
__global__ void __launch_bounds__(256) fx_plan_near(int64_t m, int nstages, const FxStage* __restrict__ stages,
                                                    const double4* __restrict__ tiles,
                                                    const double* __restrict__ records,
                                                    const double* __restrict__ tc, const double* __restrict__ tn,
                                                    const double* __restrict__ sc, const double* __restrict__ sn,
                                                    const double* __restrict__ weights, double k,
                                                    double* __restrict__ cut2, FxNear near) {
  using SH = FxShape<PDE, KIND>;
  constexpr unsigned kAll = 0xffffffffu;
  const int64_t row = blockIdx.x * (int64_t)8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= m) return;
  const double x0 = tc[3 * row], x1 = tc[3 * row + 1], x2 = tc[3 * row + 2];
  auto better = [&](double& d, int& i) {  // the least over the warp, the first of equals
    for (int o = 16; o > 0; o >>= 1) {
      const double od = __shfl_xor_sync(kAll, d, o);
      const int oi = __shfl_xor_sync(kAll, i, o);
      if (od < d || (od == d && oi < i)) {
        d = od;
        i = oi;
      }
    }
  };
  auto source2 = [&](int s, int j) {
    const double* y = records + ((int64_t)s * SH::J + j) * FX_REC;
    return fx_dist2(x0 - y[0], x1 - y[1], x2 - y[2]);
  };
  double dn = INFINITY;
  int at = 0;
#pragma unroll 4
  for (int s = lane; s < nstages; s += 32) {
    const double4 t = tiles[s];
    const double d = fx_dist2(x0 - t.x, x1 - t.y, x2 - t.z);
    if (d < dn) {
      dn = d;
      at = s;
    }
  }
  better(dn, at);
  double ds = INFINITY;
  int js = 0;
  for (int j = lane; j < stages[at].count; j += 32) {
    const double d = source2(at, j);
    if (d < ds) {
      ds = d;
      js = j;
    }
  }
  better(ds, js);
  double cut = kNearFill * weights[stages[at].src0 + js];
  int total = 0;
  // where more than kNear sources lie that close: a smaller distance, at last none
  for (int attempt = 0;; ++attempt) {
    if (!(cut > kSamePointTol2) || attempt == 8) {
      cut = kSamePointTol2;
      total = 0;
      break;
    }
    total = 0;
    const double r = sqrt(cut);
#pragma unroll 4
    for (int b = 0; b < nstages; b += 32) {
      bool want = false;
      if (b + lane < nstages) {
        const double4 t = tiles[b + lane];
        const double rr = (r + t.w) * (1 + 1e-9);
        want = fx_dist2(x0 - t.x, x1 - t.y, x2 - t.z) <= rr * rr;
      }
      for (unsigned w = __ballot_sync(kAll, want); w; w &= w - 1) {
        const int s = b + __ffs(w) - 1, cnt = stages[s].count;
        for (int j0 = 0; j0 < cnt; j0 += 32) {
          const int j = j0 + lane;
          bool take = false;
          if (j < cnt) {
            const double d2 = source2(s, j);
            take = d2 > kSamePointTol2 && d2 <= cut;
          }
          const unsigned mask = __ballot_sync(kAll, take);
          const int e = total + __popc(mask & ((1u << lane) - 1));
          if (take && e < kNear) near.idx[e * near.estep + row * near.rstep] = (int32_t)(stages[s].src0 + j);
          total += __popc(mask);
        }
      }
    }
    if (total <= kNear) break;
    cut *= 0.8 * kNear / total;
  }
  if (lane == 0) {
    cut2[row] = cut;
    near.count[row] = total;
  }
  __syncwarp();
  const double x[3] = {x0, x1, x2}, nx[3] = {tn[3 * row], tn[3 * row + 1], tn[3 * row + 2]};
  for (int e = lane; e < total; e += 32) {
    const int64_t o = e * near.estep + row * near.rstep, j = near.idx[o];
    fx_near_values<PDE, KIND>(x, nx, sc + 3 * j, sn + 3 * j, weights[j], k, near.val + o * SH::NA);
  }
}

// Scale of each target row: a bound of its kernel values.  One warp per four
// consecutive rows, which lie close together: it takes the values of their
// nearest tiles, then of every tile whose values may exceed one of the bounds
// so far (|K| from the distance to the tile alone); the others add nothing to
// the maximum.  (One thread per row left the device almost empty, 4.0 ms at
// 13,872 rows; one warp per row read the tiles 43,200 times, 2.1 ms there.
// Eight, four and two rows per warp, Theta: 43,200 complex rows 704, 668 and
// 1,121 us, 10,800 real rows of the derivative form 211, 165 and 124.)
constexpr int kPlanRows = 4;

template <int PDE, int KIND>
__global__ void __launch_bounds__(256) fx_plan_rows(int nrb, const FxRows* __restrict__ rows,
                                                    const double* __restrict__ tc, const double* __restrict__ tn,
                                                    const FxStage* __restrict__ stages,
                                                    const double4* __restrict__ tiles,
                                                    const double* __restrict__ records, FxConst c,
                                                    const double* __restrict__ cut2, double* __restrict__ rowscale,
                                                    unsigned long long* __restrict__ meta) {
  using SH = FxShape<PDE, KIND>;
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int JL = SH::J < 32 ? SH::J : 32;  // lanes along the sources of a tile
  constexpr int RP = 32 / JL;                  // rows per pass
  constexpr int NP = kPlanRows / RP;           // passes
  static_assert(kPlanRows % RP == 0, "whole passes");
  __shared__ double sx[8][kPlanRows][9];       // x, n_x, |n_x|, reach, cut2 of a warp's rows
  const int wid = blockIdx.x * 8 + (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (wid / (FX_M / kPlanRows) >= nrb) return;
  const FxRows rb = rows[wid / (FX_M / kPlanRows)];
  const int r0 = wid % (FX_M / kPlanRows) * kPlanRows;
  if (r0 >= rb.nrows) return;
  const double snorm = __longlong_as_double((long long)meta[0]);
  double (*rx)[9] = sx[threadIdx.x >> 5];
  if (lane < kPlanRows) {
    const int64_t row = rb.row0 + min(r0 + lane, rb.nrows - 1);
    double n2 = 0.0;
    for (int q = 0; q < 3; ++q) {
      const double nq = SH::tnormal ? tn[3 * row + q] : 0.0;
      rx[lane][q] = tc[3 * row + q];
      rx[lane][3 + q] = nq;
      n2 += nq * nq;
    }
    rx[lane][6] = SH::tnormal ? sqrt(n2) : 1.0;
    rx[lane][8] = SH::near ? cut2[row] : kSamePointTol2;
  }
  __syncwarp();
  auto centre2 = [&](int q, const double4& t) {  // squared distance of row q to the tile's centre
    const double a = rx[q][0] - t.x, b = rx[q][1] - t.y, e = rx[q][2] - t.z;
    return a * a + b * b + e * e;
  };
  const int s0 = rb.stage0, s1 = rb.stage0 + rb.nstages;
  double best[NP] = {};  // of rows RP * pass + lane / JL, this lane's sources
  auto tile = [&](int s) {
    const int cnt = stages[s].count;
    for (int j = lane % JL; j < cnt; j += JL) {
      const double* y = records + ((int64_t)s * SH::J + j) * FX_REC;
      const double y0 = y[0], y1 = y[1], y2 = y[2], n0 = y[3], n1 = y[4], n2 = y[5];
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        const double* t = rx[RP * p + lane / JL];
        const double a = t[0] - y0, b = t[1] - y1, e = t[2] - y2;
        const double d2 = a * a + b * b + e * e;
        if (!(d2 > 0.99 * t[8])) continue;
        const double id = rsqrt_fast(d2);
        const double rnx = fabs(a * t[3] + b * t[4] + e * t[5]), rny = fabs(a * n0 + b * n1 + e * n2);
        const double nn = fabs(t[3] * n0 + t[4] * n1 + t[5] * n2);
        best[p] = fx_max(best[p], fx_modulus<PDE, KIND>(d2 * id, id, rnx, rny, nn, c));
      }
    }
  };
  auto bound = [&](int q) {  // the largest value of row q so far, in every lane
    double v = 0.0;
#pragma unroll
    for (int p = 0; p < NP; ++p)
      if (p == q / RP && lane / JL == q % RP) v = best[p];
    for (int o = 16; o > 0; o >>= 1) v = fx_max(v, __shfl_xor_sync(kAll, v, o));
    return v;
  };
  int last = -1;
  for (int q = 0; q < kPlanRows; ++q) {
    // (the nearest one outside of the sources taken apart, which would give no bound)
    double dn = INFINITY;
    int near = s0;
    const double inner = rx[q][8] > kSamePointTol2 ? sqrt(rx[q][8]) : -INFINITY;
    for (int s = s0 + lane; s < s1; s += 32) {
      const double4 t = tiles[s];
      const double d = centre2(q, t), out = inner + t.w;
      if (d < dn && (!SH::near || out < 0.0 || d > out * out)) {
        dn = d;
        near = s;
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double d = __shfl_xor_sync(kAll, dn, o);
      const int s = __shfl_xor_sync(kAll, near, o);
      if (d < dn || (d == dn && s < near)) {
        dn = d;
        near = s;
      }
    }
    if (near != last) tile(near);
    last = near;
  }
  // Sources at least `reach` away cannot exceed the bound: the crude bound
  // falls with the distance, so the first of 64 distances (powers of sqrt 2,
  // two per lane) at which it is low enough will do.  Kept with the row.
  for (int q = 0; q < kPlanRows; ++q) {
    const double cur = bound(q), tnorm = rx[q][6], unit = tiles[last].w + sqrt(centre2(q, tiles[last]));
    double reach = INFINITY;
    for (int h = 1; h >= 0; --h) {
      const double d = exp2(0.5 * (lane + 32 * h) - 24.0) * unit;
      const unsigned ok =
          __ballot_sync(kAll, fx_modulus<PDE, KIND>(d, 1.0 / d, d * tnorm, d * snorm, tnorm * snorm, c) <= cur);
      if (ok) reach = __shfl_sync(kAll, d, __ffs(ok) - 1);
    }
    if (lane == 0) rx[q][7] = reach;
  }
  __syncwarp();
  for (int b = s0; b < s1; b += 32) {
    const int s = b + lane;
    bool want = false;
    if (s < s1) {
      const double4 t = tiles[s];
#pragma unroll
      for (int q = 0; q < kPlanRows; ++q) {
        const double rr = (rx[q][7] + t.w) * (1 + 1e-9);
        want |= centre2(q, t) < rr * rr;
      }
    }
    for (unsigned m = __ballot_sync(kAll, want); m; m &= m - 1) tile(b + __ffs(m) - 1);
  }
  for (int q = 0; q < kPlanRows; ++q) {
    const double v = bound(q) * (1 + 1e-9);  // the values' own rounding
    if (lane == 0 && r0 + q < rb.nrows) {
      if (!fx_fits(v)) atomicExch(meta + 1, 1ULL);  // NaN too
      rowscale[rb.row0 + r0 + q] = fx_fits(v) ? fx_scale(v) : 0.0;
    }
  }
}

// ---------------------------------------------------------------------------
// densities: column bounds and digit blocks
// ---------------------------------------------------------------------------
// colmax[surf * ncol + c]: bits of max |w x| over the (Re, Im) parts of column c.  Non-negative doubles
// order as their bits; a NaN's exceed every number's.
// mass[stage * ncol + c]: at most the sum of |w x| (the larger part) over the
// stage without its largest term, so that it holds for a target that is one
// of the stage's nodes, too.
constexpr int kMaxRun = 2;  // stages per warp (eight, one after another: 11 us at 1,728 nodes, two 5)

__device__ __forceinline__ double fx_mass(double sum, double top) { return fmax(0.0, (sum - top) - 1e-14 * sum); }

template <bool CPLX>
__global__ void fx_colmax(int nstages, const FxStage* __restrict__ stages, const double* __restrict__ w,
                          const double* __restrict__ x, int64_t ldx, int ncol, unsigned long long* colmax,
                          double* __restrict__ mass) {
  pdl_trigger();
  pdl_wait();
  const int run = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int s0 = run * kMaxRun, s1 = min(nstages, s0 + kMaxRun);
  for (int c = blockIdx.y; c < ncol; c += gridDim.y) {  // (a grid dimension holds 65,535)
    unsigned long long best = 0;
    int surf = -1;
    auto flush = [&]() {
      if (lane == 0 && surf >= 0) atomicMax(&colmax[(int64_t)surf * ncol + c], best);
      best = 0;
    };
    for (int s = s0; s < s1; ++s) {
      const FxStage st = stages[s];
      if (st.surf != surf) {
        flush();
        surf = st.surf;
      }
      double sum = 0.0;
      unsigned long long top = 0;
      for (int j = lane; j < st.count; j += 32) {
        const int64_t i = st.src0 + j;
        const int64_t q = (int64_t)c * ldx + i;
        double m;
        if (CPLX) {
          const double2 v = reinterpret_cast<const double2*>(x)[q];
          const double re = fabs(w[i] * v.x), im = fabs(w[i] * v.y);
          m = re > im || re != re ? re : im;
        } else {
          m = fabs(w[i] * x[q]);
        }
        sum += m;
        const unsigned long long b = (unsigned long long)__double_as_longlong(m);
        top = b > top ? b : top;
      }
      for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, top, o);
        top = other > top ? other : top;
      }
      if (lane == 0) mass[(int64_t)s * ncol + c] = fx_mass(sum, __longlong_as_double((long long)top));
      best = top > best ? top : best;
    }
    flush();
  }
}

// ---------------------------------------------------------------------------
// what the fixed-point form may take
// ---------------------------------------------------------------------------
// At most the modulus of the kernel's values (FX_THETA, FX_THETA_D: of the two
// kernels) at distance d, without the cosines of r with the normals: the size
// at which their evaluation rounds, |n| d in the place of |r.n|.  Falls with d.
template <int PDE, int KIND>
__device__ __forceinline__ double2 fx_least(double d, double nx, double ny, const FxConst& c) {
  const double id = 1.0 / d;
  const double f = (PDE == HELMHOLTZ ? sqrt(fma(c.k, c.k, id * id)) : id) * id;  // |1/d - ik|/d
  if (KIND == SL) return make_double2(id, 0.0);
  if (KIND == DL) return make_double2(f * ny, 0.0);
  if (KIND == ADL) return make_double2(f * nx, 0.0);
  if (KIND == HS) return make_double2(f * id * nx * ny, 0.0);
  if (KIND == CF) return make_double2(hypot(c.c1r, c.c1i) * f * ny + hypot(c.c2r, c.c2i) * id, 0.0);
  if (KIND == FX_THETA) return make_double2(id, f * ny);
  return make_double2(f * nx, f * id * nx * ny);
}

struct FxGuard {
  const FxRows* rows;
  const double4* tiles;
  const double* least_normal;
  const double* tcoords;
  const double* tnormals;
  const double* rowscale;
  const double* mass;   // Theta: of g1, then of g0
  int64_t mass_stride;  // between the two
  const unsigned long long* colmax;
  const unsigned long long* meta;
  int ncol;
  FxConst c;
  int* flag;
};

// Sets the flag when a row or column bound does not fit, and when a result
// would not come out as well as an FP64 sum.  What the digits leave out and
// the rounding to integers is at most 2^65.2 units per real product, a unit
// being 1/(pa pb) for the scales of the row and the column (seven products of
// order 8 of at most 2^14 each, and half a unit of either factor), so it stays
// below n 2^-52.8 T for n products while
//
//     T = sum_j S_ij |w_j x_jc| >= 2^-8 2^126 / (pa pb)
//
// (2^63/pa and 2^63/pb lie between one and 2.1 times the largest |K_ij| and
// |w_j x_jc|; S_ij is |K_ij| with |r||n| in the place of |r.n|, the size at
// which the evaluation of r.n rounds, in any form of the product).  As terms of mean zero they come to about sqrt(n) 2^-56 T at that
// limit.
//
// T is bounded from below stage by stage: the stage's mass times the kernel's
// modulus at the largest distance between its sources and the 16 rows of a
// group, from the nearest 64 stages on; a block is done when its rows and
// columns (128 x 64) have what they need.  Smooth densities need one round:
// 16 us of 1,880 at 13,872 nodes and 64 complex columns, 30 of 16,000 for the
// Theta of 43,200 nodes.
constexpr double kFxFloor = 1.0 / 256;
constexpr int kGuardRows = 16, kGuardGroups = FX_M / kGuardRows;

template <int PDE, int KIND>
__global__ void __launch_bounds__(256) fx_guard(FxGuard a) {
  pdl_trigger();
  pdl_wait();
  using SH = FxShape<PDE, KIND>;
  constexpr int NM = SH::theta ? 2 : 1, CH = 64;
  constexpr double kDown = 1.0 / 9223372036854775808.0;  // 2^-63
  __shared__ double grp[kGuardGroups][6];                // centre, radius, scale (0: nothing to check), least |n_x|
  __shared__ float m[NM][kGuardGroups][CH];
  __shared__ unsigned long long near;
  const int tid = threadIdx.x, lane = tid & 31;
  const FxRows rb = a.rows[blockIdx.x];
  if (tid == 0) near = ~0ULL;
  if (tid < FX_M) {
    const bool in = tid < rb.nrows;
    const int64_t row = rb.row0 + min(tid, rb.nrows - 1);
    double lo[3], hi[3], n2 = 0.0, p = in ? a.rowscale[row] : 0.0;
    for (int c = 0; c < 3; ++c) {
      lo[c] = hi[c] = a.tcoords[3 * row + c];
      if (SH::tnormal) n2 += a.tnormals[3 * row + c] * a.tnormals[3 * row + c];
    }
    if (p == 0.0) p = INFINITY;  // a row of zeros (or past the end)
    for (int o = kGuardRows / 2; o > 0; o >>= 1) {
      for (int c = 0; c < 3; ++c) {
        lo[c] = fmin(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
        hi[c] = fmax(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
      }
      n2 = fmin(n2, __shfl_xor_sync(0xffffffffu, n2, o));
      p = fmin(p, __shfl_xor_sync(0xffffffffu, p, o));
    }
    if (lane % kGuardRows == 0) {
      const double x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
      double* g = grp[tid / kGuardRows];
      for (int c = 0; c < 3; ++c) g[c] = (lo[c] + hi[c]) / 2;
      g[3] = 0.5 * sqrt(x * x + y * y + z * z);
      g[4] = p < INFINITY ? p : 0.0;
      g[5] = sqrt(n2);
    }
  }
  const int c = blockIdx.y * CH + (tid & (CH - 1)), g0 = tid / CH * 2;  // this thread's column and two groups
  double pb = 0.0;
  bool bad = a.meta[1] != 0;
  if (c < a.ncol) {
    const double top = __longlong_as_double((long long)a.colmax[(int64_t)rb.surf * a.ncol + c]);
    bad |= !fx_fits(top);
    if (!bad) pb = fx_scale(top);
  }
  const bool stop = tid == 0 && *(volatile int*)a.flag != 0;  // another block's finding
  if (__syncthreads_or(bad || stop)) {
    if (bad) *a.flag = 1;
    return;
  }
  const int nch = (rb.nstages + CH - 1) / CH;
  unsigned long long mine = ~0ULL;
  for (int s = tid; s < rb.nstages; s += 256) {  // the stage nearest to the first group
    const double4 t = a.tiles[rb.stage0 + s];
    const float x = (float)(grp[0][0] - t.x), y = (float)(grp[0][1] - t.y), z = (float)(grp[0][2] - t.z);
    mine = min(mine, (unsigned long long)__float_as_uint(x * x + y * y + z * z) << 32 | (unsigned)s);
  }
  for (int o = 16; o > 0; o >>= 1) mine = min(mine, __shfl_xor_sync(0xffffffffu, mine, o));
  if (lane == 0) atomicMin(&near, mine);
  __syncthreads();
  const int first = (int)((unsigned)near / CH);
  const bool need[2] = {pb > 0.0 && grp[g0][4] > 0.0, pb > 0.0 && grp[g0 + 1][4] > 0.0};
  float t[2] = {0.f, 0.f};
  for (int q = 0; q < nch; ++q) {
    const int s0 = (first + q) % nch * CH, cnt = min(CH, rb.nstages - s0);
    __syncthreads();
    for (int e = tid; e < kGuardGroups * cnt; e += 256) {
      const int g = e / cnt, s = e - g * cnt;
      const double4 tl = a.tiles[rb.stage0 + s0 + s];
      const double x = grp[g][0] - tl.x, y = grp[g][1] - tl.y, z = grp[g][2] - tl.z;
      const double d = (sqrt(x * x + y * y + z * z) + tl.w + grp[g][3]) * (1 + 1e-9);
      const double2 v = fx_least<PDE, KIND>(d, grp[g][5], a.least_normal[rb.stage0 + s0 + s], a.c);
      m[0][g][s] = (float)fmin(v.x * grp[g][4] * kDown, 1e30);
      if (SH::theta) m[NM - 1][g][s] = (float)fmin(v.y * grp[g][4] * kDown, 1e30);
    }
    __syncthreads();
    if (need[0] || need[1]) {
      const double* ms = a.mass + (int64_t)(rb.stage0 + s0) * a.ncol + c;
#pragma unroll 16
      for (int s = 0; s < cnt; ++s) {
        const float w = (float)(ms[(int64_t)s * a.ncol] * (pb * kDown));
        t[0] = fmaf(m[0][g0][s], w, t[0]);
        t[1] = fmaf(m[0][g0 + 1][s], w, t[1]);
        if (SH::theta) {
          const float u = (float)(ms[a.mass_stride + (int64_t)s * a.ncol] * (pb * kDown));
          t[0] = fmaf(m[NM - 1][g0][s], u, t[0]);
          t[1] = fmaf(m[NM - 1][g0 + 1][s], u, t[1]);
        }
      }
    }
    const bool pass = (!need[0] || t[0] >= (float)(kFxFloor * 1.001)) && (!need[1] || t[1] >= (float)(kFxFloor * 1.001));
    if (__syncthreads_and(pass)) return;
  }
  if (tid == 0) *a.flag = 1;
}

// Mean of the digit products that are dropped, p + q > 7, of a column in units
// of 256^7: A's lower digits are about 127.5 on average, so it is 1/2 times the
// sum of B's digits 1 to 7 (fx_pack), and what is left has mean zero.  Without
// it they add up where B's digits are alike: the sum of 1,536 terms of a
// constant density, largest kernel value 50 times the mean, 1.8e-16 -> 8e-18 of
// the sum (from the digits in exact arithmetic).  A sum that is exactly zero
// (kernel values of zero) stays.
__device__ __forceinline__ double fx_mean(double sum, long long digits) {
  return sum != 0.0 ? fma(0.5, (double)digits, sum) : 0.0;
}
// Sum of the digits 1 to 7 of four values.
__device__ __forceinline__ int fx_low(const uint32_t (&w)[FX_D]) {
  int s = 0;
#pragma unroll
  for (int q = 1; q < FX_D; ++q) s = __dp4a((int)w[q], 0x01010101, s);
  return s;
}
// Adds a thread's sums for column c (r, and i of complex columns) to the
// columns' totals of its surface: integers, in any order.  The threads of the
// block's first surface meet in shared memory (zero at the start).
template <int COMPS>
__device__ __forceinline__ void fx_add(int* block, bool live, int surf, int surf0, int64_t stride, int c, int r, int i,
                                       int columns, long long* total) {
  auto global = [&](int64_t at, int v) {
    atomicAdd(reinterpret_cast<unsigned long long*>(total + at), (unsigned long long)(long long)v);
  };
  if (live && surf == surf0) {
    atomicAdd(block + COMPS * c, r);
    if (COMPS == 2) atomicAdd(block + COMPS * c + 1, i);
  } else if (live) {
    global(surf * stride + COMPS * c, r);
    if (COMPS == 2) global(surf * stride + COMPS * c + 1, i);
  }
  __syncthreads();
  if ((int)threadIdx.x < COMPS * columns) global(surf0 * stride + threadIdx.x, block[threadIdx.x]);
}

// Digit blocks: stage s, digit q of column n at [chunk][q * nc + n][16 bytes].
// One thread per (chunk of a stage, column c of a plane).  A chunk holds
// groups of four sources, each value 0, then value 1; complex columns
// (2c, 2c + 1) have values (Re x, -Im x) and (Im x, Re x).
template <bool CPLX>
__global__ void fx_pack(int nstages, const FxStage* __restrict__ stages, const double* __restrict__ w,
                        const double* __restrict__ x, int64_t ldx, int c0, int ncol, int half, int nall, int nc,
                        const unsigned long long* __restrict__ colmax, const int* __restrict__ flag,
                        unsigned char* __restrict__ out, long long* __restrict__ digits) {
  pdl_trigger();
  pdl_wait();
  constexpr int JT = CPLX ? 8 : 16;  // sources of a chunk
  // plane blockIdx.y: columns c0 + y * half and on
  c0 += blockIdx.y * half;
  ncol = min(half, ncol - (int)blockIdx.y * half);
  out += (size_t)blockIdx.y * nstages * nc * (FX_D * FX_K);
  const int per = CPLX ? nc / 2 : nc;
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int c = (int)(id % per), chunk = (int)(id / per % 4);
  const int64_t s = id / per / 4;
  if (*flag) return;
  __shared__ int low[FX_NMAX];
  if (threadIdx.x < FX_NMAX) low[threadIdx.x] = 0;
  __syncthreads();
  const bool in = s < nstages;
  const FxStage st = stages[in ? s : nstages - 1];
  const bool live = in && c < ncol;
  const double p =
      live ? fx_scale(__longlong_as_double((long long)colmax[(int64_t)st.surf * nall + c0 + c])) : 0.0;
  uint4* o = reinterpret_cast<uint4*>(out + s * ((int64_t)nc * FX_D * FX_K) + (int64_t)chunk * (nc * FX_D * 16));
  uint32_t re[JT / 4][FX_D], im[CPLX ? 2 : 1][FX_D], mi[CPLX ? 2 : 1][FX_D];
#pragma unroll
  for (int h = 0; h < JT / 4; ++h) {
    uint2 a[4], b[4], m[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = chunk * JT + 4 * h + e;
      double vr = 0.0, vi = 0.0;
      if (live && j < st.count) {
        const int64_t i = st.src0 + j, q = (int64_t)(c0 + c) * ldx + i;
        if (CPLX) {
          const double2 v = reinterpret_cast<const double2*>(x)[q];
          vr = w[i] * v.x;
          vi = w[i] * v.y;
        } else {
          vr = w[i] * x[q];
        }
      }
      a[e] = fx_digits(vr * p);
      if (CPLX) {
        b[e] = fx_digits(vi * p);
        m[e] = fx_digits(-vi * p);
      }
    }
    fx_pack4(a, re[h]);
    if constexpr (CPLX) {
      fx_pack4(b, im[h]);
      fx_pack4(m, mi[h]);
    }
  }
  int lr = 0, li = 0, lm = 0;
#pragma unroll
  for (int h = 0; h < JT / 4; ++h) {
    lr += fx_low(re[h]);
    if constexpr (CPLX) {
      li += fx_low(im[h]);
      lm += fx_low(mi[h]);
    }
  }
  constexpr int COMPS = CPLX ? 2 : 1;
  fx_add<COMPS>(low, live, st.surf, stages[blockIdx.x * (int64_t)blockDim.x / per / 4].surf, (int64_t)nall * COMPS, c,
                lr + lm, li + lr, ncol, digits + (int64_t)c0 * COMPS);
  if (!in) return;
#pragma unroll
  for (int q = 0; q < FX_D; ++q) {
    if constexpr (CPLX) {
      o[q * nc + 2 * c] = make_uint4(re[0][q], mi[0][q], re[1][q], mi[1][q]);
      o[q * nc + 2 * c + 1] = make_uint4(im[0][q], re[0][q], im[1][q], re[1][q]);
    } else {
      o[q * nc + c] = make_uint4(re[0][q], re[1][q], re[2][q], re[3][q]);
    }
  }
}

// Y += alpha * (1/(4 pi)) * (sources taken apart) for four columns of a row,
// four threads per row with a quarter of the entries each.  Bound by the
// gathers of the densities (13,872 rows, 64 complex columns: 71 us of 2,115);
// one thread per row left few in flight (1,728 rows 36 us, now 16).
template <bool CPLX>
__global__ void fx_near_add(int64_t m, FxNear near, const double* __restrict__ x, int64_t ldx, double* y, int64_t ldy,
                            int c0, int ncol, double ar, double ai, const int* __restrict__ flag) {
  pdl_trigger();
  pdl_wait();
  constexpr int U = 4;
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, row = min(id / 4, m - 1);
  const int f = blockIdx.y * U;
  if (*flag) return;
  double sr[U] = {}, si[U] = {};
  const int cnt = near.count[row];
  const double* xc[U];
#pragma unroll
  for (int u = 0; u < U; ++u) xc[u] = x + (int64_t)(c0 + min(f + u, ncol - 1)) * ldx * (CPLX ? 2 : 1);
#pragma unroll 4
  for (int e = id & 3; e < cnt; e += 4) {
    const int64_t o = e * near.estep + row * near.rstep, j = near.idx[o];
    const double2 v = CPLX ? reinterpret_cast<const double2*>(near.val)[o] : make_double2(near.val[o], 0.0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (CPLX) {
        const double2 t = reinterpret_cast<const double2*>(xc[u])[j];
        sr[u] = fma(v.x, t.x, fma(-v.y, t.y, sr[u]));
        si[u] = fma(v.x, t.y, fma(v.y, t.x, si[u]));
      } else {
        sr[u] = fma(v.x, xc[u][j], sr[u]);
      }
    }
  }
  constexpr double kScale = 1.0 / (4 * kPi);
  double vr = 0.0, vi = 0.0;
#pragma unroll
  for (int u = 0; u < U; ++u) {  // the row's sum of column u to its thread u
    double r = sr[u], i = si[u];
    for (int o = 2; o > 0; o >>= 1) {
      r += __shfl_xor_sync(0xffffffffu, r, o);
      if (CPLX) i += __shfl_xor_sync(0xffffffffu, i, o);
    }
    if ((id & 3) == u) {
      vr = kScale * r;
      vi = kScale * i;
    }
  }
  const int c = f + (int)(id & 3);
  if (id / 4 >= m || c >= ncol) return;
  const int64_t q = (int64_t)(c0 + c) * ldy + row;
  if (CPLX) {
    double2* Y = reinterpret_cast<double2*>(y);
    double2 t = Y[q];
    t.x += ar * vr - ai * vi;
    t.y += ar * vi + ai * vr;
    Y[q] = t;
  } else {
    y[q] += ar * vr;
  }
}

// The same for Theta: out[row, k] += 1/(4 pi) sum (ADL w g1 - HS w g0).
template <bool CPLX>
__global__ void fx_near_theta(int64_t m, int ns, FxNear near, const double2* __restrict__ g0,
                              const double2* __restrict__ g1, double2* out, const int* __restrict__ flag) {
  pdl_trigger();
  pdl_wait();
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, row = id / ns;
  const int k = (int)(id - row * ns);
  if (row >= m || *flag) return;
  double sr = 0.0, si = 0.0;
  const int cnt = near.count[row];
#pragma unroll 8
  for (int e = 0; e < cnt; ++e) {
    const int64_t o = e * near.estep + row * near.rstep, j = near.idx[o];
    const double2 a = g1[j * ns + k], b = g0[j * ns + k];
    if (CPLX) {
      const double2 s = reinterpret_cast<const double2*>(near.val)[2 * o], d = reinterpret_cast<const double2*>(near.val)[2 * o + 1];
      sr = fma(s.x, a.x, fma(-s.y, a.y, sr));
      si = fma(s.x, a.y, fma(s.y, a.x, si));
      sr = fma(-d.x, b.x, fma(d.y, b.y, sr));
      si = fma(-d.x, b.y, fma(-d.y, b.x, si));
    } else {
      sr = fma(near.val[2 * o], a.x, sr);
      sr = fma(-near.val[2 * o + 1], b.x, sr);
    }
  }
  constexpr double kScale = 1.0 / (4 * kPi);
  double2 v = out[id];
  v.x = fma(kScale, sr, v.x);
  v.y = fma(kScale, si, v.y);
  out[id] = v;
}

// Theta: column bounds over the traces (both arrays share a column's scale,
// since their products share the accumulators) and the masses of g1 and g0.
// One thread per (stage, column).
__global__ void fx_theta_max(int nstages, const FxStage* __restrict__ stages, int ns, bool cplx,
                             const double* __restrict__ w, const double2* __restrict__ g0,
                             const double2* __restrict__ g1, unsigned long long* colmax, double* __restrict__ mass) {
  pdl_trigger();
  pdl_wait();
  __shared__ unsigned long long best[32];
  if (threadIdx.x < 32) best[threadIdx.x] = 0;
  __syncthreads();
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int s = (int)(id / ns), k = (int)(id - (int64_t)s * ns);
  if (s < nstages) {
    const FxStage st = stages[s];
    double sum[2] = {0.0, 0.0};
    unsigned long long top[2] = {0, 0};
    for (int j = 0; j < st.count; ++j) {
      const int64_t i = st.src0 + j, e = i * ns + k;
      const double wj = w[i];
      const double2 v[2] = {g1[e], g0[e]};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const double re = fabs(wj * v[q].x), im = cplx ? fabs(wj * v[q].y) : 0.0;
        const double mx = re > im || re != re ? re : im;
        const unsigned long long b = (unsigned long long)__double_as_longlong(mx);
        sum[q] += mx;
        top[q] = b > top[q] ? b : top[q];
      }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q)
      mass[(int64_t)q * nstages * ns + id] = fx_mass(sum[q], __longlong_as_double((long long)top[q]));
    atomicMax(&best[k], top[0] > top[1] ? top[0] : top[1]);
  }
  __syncthreads();
  if ((int)threadIdx.x < ns) atomicMax(&colmax[threadIdx.x], best[threadIdx.x]);
}

// Digit blocks of the traces: values (S; D), complex (Sr, Si; Dr, Di), against
// (g1; -g0), complex columns (Re, Im): (g1r, g1i), (-g1i, g1r), (-g0r, -g0i),
// (g0i, -g0r).
template <bool CPLX>
__global__ void fx_theta_pack(int nstages, const FxStage* __restrict__ stages, const double* __restrict__ w,
                              const double2* __restrict__ g0, const double2* __restrict__ g1, int ns, int nc,
                              const unsigned long long* __restrict__ colmax, const int* __restrict__ flag,
                              unsigned char* __restrict__ out, long long* __restrict__ digits) {
  pdl_trigger();
  pdl_wait();
  constexpr int JT = CPLX ? 4 : 8;
  const int per = CPLX ? nc / 2 : nc;
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int c = (int)(id % per), chunk = (int)(id / per % 4);
  const int64_t s = id / per / 4;
  if (*flag) return;
  __shared__ int low[FX_NMAX];
  if (threadIdx.x < FX_NMAX) low[threadIdx.x] = 0;
  __syncthreads();
  const bool in = s < nstages;
  const FxStage st = stages[in ? s : nstages - 1];
  const bool live = in && c < ns;
  const double p = live ? fx_scale(__longlong_as_double((long long)colmax[c])) : 0.0;
  uint4* o = reinterpret_cast<uint4*>(out + s * ((int64_t)nc * FX_D * FX_K) + (int64_t)chunk * (nc * FX_D * 16));
  double2 a[JT], b[JT];
#pragma unroll
  for (int e = 0; e < JT; ++e) {
    const int j = chunk * JT + e;
    a[e] = b[e] = make_double2(0.0, 0.0);
    if (live && j < st.count) {
      const int64_t i = st.src0 + j, q = i * ns + c;
      const double wj = w[i];
      const double2 u = g0[q], v = g1[q];
      a[e] = make_double2(wj * u.x, wj * u.y);
      b[e] = make_double2(wj * v.x, wj * v.y);
    }
  }
  auto pack = [&](auto get, uint32_t (&wd)[FX_D]) {
    uint2 d[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) d[e] = fx_digits(get(e) * p);
    fx_pack4(d, wd);
  };
  uint32_t wd[CPLX ? 6 : 4][FX_D];
  if constexpr (CPLX) {
    pack([&](int e) { return b[e].x; }, wd[0]);
    pack([&](int e) { return b[e].y; }, wd[1]);
    pack([&](int e) { return -b[e].y; }, wd[2]);
    pack([&](int e) { return -a[e].x; }, wd[3]);
    pack([&](int e) { return -a[e].y; }, wd[4]);
    pack([&](int e) { return a[e].y; }, wd[5]);
    fx_add<2>(low, live, 0, 0, 0, c, fx_low(wd[0]) + fx_low(wd[2]) + fx_low(wd[3]) + fx_low(wd[5]),
              fx_low(wd[1]) + fx_low(wd[0]) + fx_low(wd[4]) + fx_low(wd[3]), ns, digits);
    if (!in) return;
#pragma unroll
    for (int q = 0; q < FX_D; ++q) {
      o[q * nc + 2 * c] = make_uint4(wd[0][q], wd[2][q], wd[3][q], wd[5][q]);
      o[q * nc + 2 * c + 1] = make_uint4(wd[1][q], wd[0][q], wd[4][q], wd[3][q]);
    }
  } else {
    pack([&](int e) { return b[e].x; }, wd[0]);
    pack([&](int e) { return b[e + 4].x; }, wd[1]);
    pack([&](int e) { return -a[e].x; }, wd[2]);
    pack([&](int e) { return -a[e + 4].x; }, wd[3]);
    fx_add<1>(low, live, 0, 0, 0, c, fx_low(wd[0]) + fx_low(wd[1]) + fx_low(wd[2]) + fx_low(wd[3]), 0, ns, digits);
    if (!in) return;
#pragma unroll
    for (int q = 0; q < FX_D; ++q) o[q * nc + c] = make_uint4(wd[0][q], wd[2][q], wd[1][q], wd[3][q]);
  }
}

// ---------------------------------------------------------------------------
// results
// ---------------------------------------------------------------------------
// Sum of the slots of (row block, real column), unscaled.
__device__ __forceinline__ double fx_total(const FxRows& rb, const double* __restrict__ partial, int nc, int col,
                                           int r) {
  double s = 0.0;
  for (int q = 0; q < rb.nseg; ++q) s += partial[((size_t)(rb.slot0 + q) * nc + col) * FX_M + r];
  return s;
}

constexpr double kFxUnit = 72057594037927936.0;  // 256^7

// 1/p for a power of two p (0 for 0)
__device__ __forceinline__ double fx_inverse(double p) {
  return p > 0.0 ? __longlong_as_double((2046LL << 52) - __double_as_longlong(p)) : 0.0;
}

struct FxOut {
  const FxRows* rows;
  const double* partial;
  const double* rowscale;
  const unsigned long long* colmax;
  const long long* digits;
  const int* flag;
  const int64_t* rowptr;  // correction, null when there is none
  const int32_t* col;
  const double* val;
  const double* x;
  double* y;
  int64_t ldx, ldy;
  int c0, nall, nc, half, nslots;  // half: columns per plane
  double scale, ar, ai, br, bi;
  bool beta_zero;
};

template <bool CPLX>
__global__ void __launch_bounds__(FX_M) fx_finish(FxOut o) {
  pdl_trigger();
  pdl_wait();
  if (*o.flag) return;
  const FxRows rb = o.rows[blockIdx.x];
  const int r = threadIdx.x, c = blockIdx.y, cg = o.c0 + c;
  if (r >= rb.nrows) return;
  const int64_t row = rb.row0 + r;
  const double pb = fx_scale(__longlong_as_double((long long)o.colmax[(int64_t)rb.surf * o.nall + cg]));
  // sums are in units of 256^7 / (pa pb)
  const double u = fx_inverse(o.rowscale[row]) * fx_inverse(pb) * (o.scale * kFxUnit);
  const double* partial = o.partial + (size_t)(c / o.half) * o.nslots * o.nc * FX_M;
  const int cp = c % o.half;
  double sr, si = 0.0;
  const long long* d = o.digits + ((int64_t)rb.surf * o.nall + cg) * (CPLX ? 2 : 1);
  if (CPLX) {
    sr = u * fx_mean(fx_total(rb, partial, o.nc, 2 * cp, r), d[0]);
    si = u * fx_mean(fx_total(rb, partial, o.nc, 2 * cp + 1, r), d[1]);
  } else {
    sr = u * fx_mean(fx_total(rb, partial, o.nc, cp, r), d[0]);
  }
  if (o.rowptr) {
    for (int64_t p = o.rowptr[row]; p < o.rowptr[row + 1]; ++p) {
      const int64_t j = (int64_t)cg * o.ldx + o.col[p];
      if (CPLX) {
        const double2 v = reinterpret_cast<const double2*>(o.val)[p], xv = reinterpret_cast<const double2*>(o.x)[j];
        sr = fma(v.x, xv.x, fma(-v.y, xv.y, sr));
        si = fma(v.x, xv.y, fma(v.y, xv.x, si));
      } else {
        sr = fma(o.val[p], o.x[j], sr);
      }
    }
  }
  const int64_t q = (int64_t)cg * o.ldy + row;
  if (CPLX) {
    double2* Y = reinterpret_cast<double2*>(o.y);
    double yr = o.ar * sr - o.ai * si, yi = o.ar * si + o.ai * sr;
    if (!o.beta_zero) {
      const double2 yo = Y[q];
      yr += o.br * yo.x - o.bi * yo.y;
      yi += o.br * yo.y + o.bi * yo.x;
    }
    Y[q] = make_double2(yr, yi);
  } else {
    double v = o.ar * sr;
    if (!o.beta_zero) v += o.br * o.y[q];
    o.y[q] = v;
  }
}

template <bool CPLX>
__global__ void __launch_bounds__(FX_M) fx_theta_finish(const FxRows* __restrict__ rows,
                                                        const double* __restrict__ partial,
                                                        const double* __restrict__ rowscale,
                                                        const unsigned long long* __restrict__ colmax,
                                                        const long long* __restrict__ digits, int ns, int nc,
                                                        const int* __restrict__ flag, double2* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  if (*flag) return;
  const FxRows rb = rows[blockIdx.x];
  const int r = threadIdx.x, c = blockIdx.y;
  if (r >= rb.nrows) return;
  const int64_t row = rb.row0 + r;
  const double u = fx_inverse(rowscale[row]) *
                   fx_inverse(fx_scale(__longlong_as_double((long long)colmax[c]))) * (1.0 / (4 * kPi) * kFxUnit);
  double2 v = make_double2(0.0, 0.0);
  if (CPLX) {
    v.x = u * fx_mean(fx_total(rb, partial, nc, 2 * c, r), digits[2 * c]);
    v.y = u * fx_mean(fx_total(rb, partial, nc, 2 * c + 1, r), digits[2 * c + 1]);
  } else {
    v.x = u * fx_mean(fx_total(rb, partial, nc, c, r), digits[c]);
  }
  out[row * ns + c] = v;
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
template <class F>
static void fx_dispatch(int pde, int kind, F&& f) {
  auto by = [&](auto pc) {
    constexpr int P = decltype(pc)::value;
    switch (kind) {
      case SL: return f(pc, std::integral_constant<int, SL>());
      case DL: return f(pc, std::integral_constant<int, DL>());
      case ADL: return f(pc, std::integral_constant<int, ADL>());
      case HS: return f(pc, std::integral_constant<int, HS>());
      case CF: return f(pc, std::integral_constant<int, CF>());
      case FX_THETA: return f(pc, std::integral_constant<int, FX_THETA>());
      default: return f(pc, std::integral_constant<int, FX_THETA_D>());
    }
    (void)P;
  };
  if (pde == HELMHOLTZ)
    by(std::integral_constant<int, HELMHOLTZ>());
  else
    by(std::integral_constant<int, LAPLACE>());
}

static FxConst fx_const(const FxProblem& p) {
  return FxConst{p.k,     p.k * FX_TAB / (2 * kPi), p.c1[0], p.c1[1], p.c2[0], p.c2[1],
                 p.k * p.c1[0], p.k * p.c1[1]};
}

const int* fx_flag(const inti_ctx* ctx) { return ctx->fx.work.as<int>(); }

void fx_hold(inti_ctx* ctx, FxPlan& plan) {
  if (plan.held) return;
  plan.held = true;
  ctx->fx.users++;
}

void fx_drop(inti_ctx* ctx, FxPlan& plan) {
  if (!plan.held) return;
  plan.held = false;
  if (--ctx->fx.users > 0) return;
  for (DevBuf* b : {&ctx->fx.bdig, &ctx->fx.partial, &ctx->fx.work, &ctx->fx.mass}) b->release();
}

// Where the contraction is the faster form.  Below about 2e6 pairs (1,400
// nodes squared) the FP64 MMA kernel's single launch is as fast: 8 complex
// columns at 1,200 nodes take 123 us either way, at 1,728 nodes 170 us against
// 64 us here (64 columns 407 against 125 us).  Theta pays for its plan (row
// bounds, work lists) every time, about 0.1 ms: real values break even near
// 5e7 pairs (7,000 nodes), complex ones near 2e7.  The derivative form adds the
// sources taken apart: real values 0.62 against 0.65 ms at 8,112 nodes, 0.78
// against 0.71 at 9,408, complex ones 0.59 against 0.66 at 4,800, 0.80 against
// 0.78 at 5,808; with more targets than sources, complex values, 2,352 x 20,000
// 2.38 both, 3,888 x 20,000 2.73 against 2.57.
// Few sources leave little of an item next to its hand-over (and a surface's
// last stage partly empty), while the FP64 MMA kernel's blocks are short then.
// Ratio of its time to the time here, 8 and 64 columns, sources x targets:
// Laplace SL 256 x 16,000 0.59 and 0.70, 512 x 8,000 0.73 and 0.76, 768 x 8,000
// 0.77 and 0.84, 1,024 x 8,000 0.98 and 1.09, 1,024 x 2,000 1.15 and 1.37, 2,048
// x 8,000 1.34 and 1.42; batches of surfaces of 216 nodes 0.63 .. 0.91, 486
// nodes 0.87 .. 1.40, 864 nodes 1.31 .. 2.12.  With sources taken apart: HS
// 1,024 x 8,000 0.76 and 0.85, 1,500 x 8,000 0.88 and 1.01, 1,452 x 1,452 1.12
// and 1.42.
bool fx_pays(int pde, int kind, double targets, double pairs) {
  if (kind < FX_THETA) return pairs >= 2e6 && pairs >= (kind == HS ? 1400.0 : 850.0) * targets;
  if (kind == FX_THETA_D) return pairs >= (pde == HELMHOLTZ ? 3.3e7 : 8.8e7) && pairs >= 3500.0 * targets;
  return pairs >= (pde == HELMHOLTZ ? 2e7 : 5e7);
}

// Columns of one pass: a multiple of eight, at least 16, at most 64.
static int fx_width(int real_columns) { return std::min(FX_NMAX, std::max(16, (real_columns + 7) / 8 * 8)); }
// The next pass over `left` columns: up to 64 real ones in one plane, up to
// 128 in two equal planes, one per CTA of a pair.
struct FxPass {
  int cols, planes, half, nc;  // columns, planes, columns per plane, real columns of a plane (padded)
};
static FxPass fx_pass(int left, int comps) {
  const int one = FX_NMAX / comps;
  FxPass p;
  p.cols = std::min(left, 2 * one);
  p.planes = p.cols > one ? 2 : 1;
  p.half = (p.cols + p.planes - 1) / p.planes;
  p.nc = fx_width(p.half * comps);
  return p;
}
// work: [flag, counter per pass (up to 63) | column bounds | digit sums of the
// columns' one or two components]
constexpr int FX_COUNTERS = 64;
static size_t fx_work_bytes(const FxProblem& p, int nsurf, int ncols) {
  return sizeof(int) * FX_COUNTERS + sizeof(long long) * (size_t)nsurf * ncols * (p.pde == HELMHOLTZ ? 3 : 2);
}

// Kernels with sources taken apart (of one surface: the first target is 0).
static bool fx_near_kind(int kind) { return kind == HS || kind == FX_THETA_D; }
static FxNear fx_near(const FxProblem& p, const FxPlan& plan) {
  const int64_t m = plan.ntargets;
  FxNear n;
  n.count = plan.near_idx.as<int32_t>();
  n.idx = n.count + m;
  n.val = plan.near_val.as<double>();
  n.estep = p.kind == HS ? m : 1;  // threads run along the rows, of Theta along a row's columns
  n.rstep = p.kind == HS ? 1 : kNear;
  return n;
}

static void fx_plan(inti_ctx* ctx, const FxProblem& p, FxPlan& plan) {
  const int J = FX_K / fx_na(p.pde, p.kind);
  const int nsurf = (int)p.row.size();
  std::vector<FxRows> rows;
  std::vector<FxItem> items;
  std::vector<FxStage> stages;
  plan.ntargets = 0;
  double total = 0.0;
  for (int s = 0; s < nsurf; ++s)
    total += (double)((p.nrow[s] + FX_M - 1) / FX_M) * (double)((p.nsrc[s] + J - 1) / J);
  // Runs of about a sixth of an SM's share of the stages (a short tail), at
  // least four stages (an item costs about one stage in hand-over).
  const int run = (int)std::max(4.0, std::ceil(total / (6.0 * ctx->num_sms)));
  plan.nslots = 0;
  for (int s = 0; s < nsurf; ++s) {
    const int stage0 = (int)stages.size(), nst = (int)((p.nsrc[s] + J - 1) / J);
    for (int t = 0; t < nst; ++t)
      stages.push_back(FxStage{p.src[s] + (int64_t)t * J, (int32_t)std::min<int64_t>(J, p.nsrc[s] - (int64_t)t * J), s});
    const int nseg = std::max(1, (nst + run - 1) / run);
    for (int64_t r = 0; r < p.nrow[s]; r += FX_M) {
      const int rb = (int)rows.size();
      rows.push_back(FxRows{p.row[s] + r, (int32_t)std::min<int64_t>(FX_M, p.nrow[s] - r), plan.nslots, nseg, s, stage0,
                            nst});
      for (int q = 0; q < nseg; ++q) {
        const int a = (int)((int64_t)nst * q / nseg), b = (int)((int64_t)nst * (q + 1) / nseg);
        items.push_back(FxItem{rb, a, b - a, plan.nslots + q});
      }
      plan.nslots += nseg;
    }
    plan.ntargets = std::max(plan.ntargets, p.row[s] + p.nrow[s]);
  }
  std::stable_sort(items.begin(), items.end(), [](const FxItem& a, const FxItem& b) { return a.nstages > b.nstages; });
  plan.nrows = (int)rows.size();
  plan.nitems = (int)items.size();
  plan.nstages = (int)stages.size();
  plan.nsurf = nsurf;
  // one upload (rows | stages | items): each copy from pageable memory waits
  // for the stream, and a correction builds its plan every time
  const size_t b_rows = sizeof(FxRows) * rows.size(), b_stages = sizeof(FxStage) * stages.size(),
               b_items = sizeof(FxItem) * items.size();
  std::vector<unsigned char> h(b_rows + b_stages + b_items);
  std::memcpy(h.data(), rows.data(), b_rows);
  std::memcpy(h.data() + b_rows, stages.data(), b_stages);
  std::memcpy(h.data() + b_rows + b_stages, items.data(), b_items);
  plan.tables.ensure(h.size());
  INTI_CUDA(cudaMemcpyAsync(plan.tables.p, h.data(), h.size(), cudaMemcpyHostToDevice, ctx->stream));
  plan.rows = plan.tables.as<FxRows>();
  plan.stages = reinterpret_cast<const FxStage*>(plan.tables.as<unsigned char>() + b_rows);
  plan.items = reinterpret_cast<const FxItem*>(plan.tables.as<unsigned char>() + b_rows + b_stages);
  plan.records.ensure(sizeof(double) * FX_REC * J * stages.size());
  plan.tiles.ensure(sizeof(double4) * stages.size());
  plan.least_normal.ensure(sizeof(double) * stages.size());
  plan.rowscale.ensure(sizeof(double) * std::max<int64_t>(plan.ntargets, 1));
  plan.meta.ensure(sizeof(unsigned long long) * 2);
  if (fx_near_kind(p.kind)) {
    plan.cut2.ensure(sizeof(double) * plan.ntargets);
    plan.near_idx.ensure(sizeof(int32_t) * plan.ntargets * (1 + kNear));
    plan.near_val.ensure(sizeof(double) * plan.ntargets * kNear * fx_na(p.pde, p.kind));
  }
  INTI_CUDA(cudaMemsetAsync(plan.meta.p, 0, sizeof(unsigned long long) * 2, ctx->stream));
  fx_plan_sources<<<(plan.nstages + 7) / 8, 256, 0, ctx->stream>>>(
      plan.nstages, J, plan.stages, p.coords, p.normals, plan.records.as<double>(),
      plan.tiles.as<double4>(), plan.least_normal.as<double>(), plan.meta.as<unsigned long long>());
  fx_dispatch(p.pde, p.kind, [&](auto pc, auto kc) {
    constexpr int P = decltype(pc)::value, K = decltype(kc)::value;
    if constexpr (FxShape<P, K>::near) {
      const int64_t m = plan.ntargets;
      fx_plan_near<P, K><<<(unsigned)((m + 7) / 8), 256, 0, ctx->stream>>>(
          m, plan.nstages, plan.stages, plan.tiles.as<double4>(), plan.records.as<double>(), p.tcoords, p.tnormals,
          p.coords, p.normals, p.weights, p.k, plan.cut2.as<double>(), fx_near(p, plan));
      ctx->launches++;
    }
    fx_plan_rows<P, K><<<(unsigned)plan.nrows * (FX_M / kPlanRows / 8), 256, 0, ctx->stream>>>(
        plan.nrows, plan.rows, p.tcoords, p.tnormals, plan.stages, plan.tiles.as<double4>(),
        plan.records.as<double>(), fx_const(p), plan.cut2.as<double>(), plan.rowscale.as<double>(),
        plan.meta.as<unsigned long long>());
    INTI_CUDA(cudaFuncSetAttribute(fx_contract_kernel<P, K, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   FxShape<P, K>::SMEM));
    if constexpr (!FxShape<P, K>::theta)
      INTI_CUDA(cudaFuncSetAttribute(fx_contract_kernel<P, K, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     FxShape<P, K>::SMEM));
  });
  ctx->launches += 2;
  INTI_CUDA(cudaGetLastError());
  if (!ctx->fx.tab.p) {
    std::vector<double2> t(FX_TAB);
    const long double d = (long double)(2.0 * kPi / FX_TAB);
    for (int m = 0; m < FX_TAB; ++m) t[m] = make_double2((double)cosl(m * d), (double)sinl(m * d));
    ctx->fx.tab.ensure(sizeof(double2) * FX_TAB);
    INTI_CUDA(cudaMemcpyAsync(ctx->fx.tab.p, t.data(), sizeof(double2) * FX_TAB, cudaMemcpyHostToDevice, ctx->stream));
  }
  plan.ready = true;
}

bool fx_prepare(inti_ctx* ctx, const FxProblem& p, FxPlan& plan, int ncols) {
  const FxPass w = fx_pass(ncols, p.pde == HELMHOLTZ ? 2 : 1);  // the widest pass
  auto digits = [&] { return (size_t)plan.nstages * w.planes * w.nc * FX_D * FX_K; };
  auto partial = [&] { return sizeof(double) * (size_t)plan.nslots * w.planes * w.nc * FX_M; };
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  INTI_CUDA(cudaStreamIsCapturing(ctx->stream, &cap));
  if (cap != cudaStreamCaptureStatusNone) return false;
  try {
    if (!plan.ready) fx_plan(ctx, p, plan);
    ctx->fx.bdig.ensure(digits());
    ctx->fx.partial.ensure(partial());
    ctx->fx.work.ensure(fx_work_bytes(p, plan.nsurf, ncols));
    ctx->fx.mass.ensure(sizeof(double) * (size_t)plan.nstages * ncols * (p.kind >= FX_THETA ? 2 : 1));
  } catch (const Error& e) {
    if (e.code != INTI_E_NOMEM) throw;
    return false;
  }
  return true;
}

static unsigned long long* fx_colmax_ptr(inti_ctx* ctx) {
  return reinterpret_cast<unsigned long long*>(ctx->fx.work.as<int>() + FX_COUNTERS);
}

static long long* fx_digits_ptr(inti_ctx* ctx, const FxPlan& plan, int ncols) {
  return reinterpret_cast<long long*>(fx_colmax_ptr(ctx)) + (size_t)plan.nsurf * ncols;
}

static void fx_guard_run(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, int ncol) {
  FxGuard a;
  a.rows = plan.rows;
  a.tiles = plan.tiles.as<double4>();
  a.least_normal = plan.least_normal.as<double>();
  a.tcoords = p.tcoords;
  a.tnormals = p.tnormals;
  a.rowscale = plan.rowscale.as<double>();
  a.mass = ctx->fx.mass.as<double>();
  a.mass_stride = (int64_t)plan.nstages * ncol;
  a.colmax = fx_colmax_ptr(ctx);
  a.meta = plan.meta.as<unsigned long long>();
  a.ncol = ncol;
  a.c = fx_const(p);
  a.flag = ctx->fx.work.as<int>();
  fx_dispatch(p.pde, p.kind, [&](auto pc, auto kc) {
    constexpr int P = decltype(pc)::value, K = decltype(kc)::value;
    launch_pdl(ctx->stream, dim3((unsigned)plan.nrows, (unsigned)((ncol + 63) / 64)), 256, 0, &fx_guard<P, K>, a);
  });
  ctx->launches++;
}

static void fx_run(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, int nc, int planes, int* counter) {
  FxArgs a;
  a.rows = plan.rows;
  a.items = plan.items;
  a.nitems = plan.nitems;
  a.nc = nc;
  a.tcoords = p.tcoords;
  a.tnormals = p.tnormals;
  a.rowscale = plan.rowscale.as<double>();
  a.cut2 = plan.cut2.as<double>();
  a.records = plan.records.as<double>();
  a.bdig = ctx->fx.bdig.as<unsigned char>();
  a.nstages = plan.nstages;
  a.nslots = plan.nslots;
  a.tab = ctx->fx.tab.as<double2>();
  a.partial = ctx->fx.partial.as<double>();
  a.c = fx_const(p);
  a.counter = counter;
  a.flag = fx_flag(ctx);
  a.err = ctx->err_flag.as<int>();
  ctx->flag_armed = true;
  fx_dispatch(p.pde, p.kind, [&](auto pc, auto kc) {
    constexpr int P = decltype(pc)::value, K = decltype(kc)::value;
    if (planes == 1) {
      launch_pdl(ctx->stream, (unsigned)std::min(ctx->num_sms, plan.nitems), FX_THREADS, FxShape<P, K>::SMEM,
                 &fx_contract_kernel<P, K, 1>, a);
    } else if constexpr (!FxShape<P, K>::theta) {
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)(2 * std::min(ctx->num_sms / 2, plan.nitems)));
      cfg.blockDim = dim3(FX_THREADS);
      cfg.dynamicSmemBytes = FxShape<P, K>::SMEM;
      cfg.stream = ctx->stream;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      INTI_CUDA(cudaLaunchKernelEx(&cfg, fx_contract_kernel<P, K, 2>, a));
    }
  });
  ctx->launches++;
  INTI_CUDA(cudaGetLastError());
}

// The kernels of a product are launched programmatically, each waiting for the
// one before it at its start: without that the check's launch cost 10 us at
// 1,728 nodes (8 columns, Laplace SL, back to the host: 66 us without the
// check, 78 with it, 56 so).
void fx_apply(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, const inti_csr* corr, const double* x,
              int64_t ldx, double* y, int64_t ldy, int nrhs, const double* alpha, const double* beta) {
  const bool cplx = p.pde == HELMHOLTZ;
  const int comps = cplx ? 2 : 1;
  INTI_CUDA(cudaMemsetAsync(ctx->fx.work.p, 0, fx_work_bytes(p, plan.nsurf, nrhs), ctx->stream));
  int* flag = ctx->fx.work.as<int>();
  unsigned long long* colmax = fx_colmax_ptr(ctx);
  const FxStage* st = plan.stages;
  auto by_type = [&](auto cc) {
    constexpr bool C = decltype(cc)::value;
    const int runs = (plan.nstages + kMaxRun - 1) / kMaxRun;
    launch_pdl(ctx->stream, dim3((runs + 7) / 8, std::min(nrhs, 65535)), 256, 0, &fx_colmax<C>, plan.nstages, st,
               p.weights, x, ldx, nrhs, colmax, ctx->fx.mass.as<double>());
    ctx->launches++;
    fx_guard_run(ctx, p, plan, nrhs);
    int pass = 0;
    FxPass w;
    for (int c0 = 0; c0 < nrhs; c0 += w.cols, ++pass) {
      w = fx_pass(nrhs - c0, comps);
      const int64_t threads = (int64_t)plan.nstages * 4 * (w.nc / comps);
      launch_pdl(ctx->stream, dim3((unsigned)((threads + 127) / 128), w.planes), 128, 0, &fx_pack<C>, plan.nstages, st,
                 p.weights, x, ldx, c0, w.cols, w.half, nrhs, w.nc, colmax, flag, ctx->fx.bdig.as<unsigned char>(),
                 fx_digits_ptr(ctx, plan, nrhs));
      ctx->launches++;
      const int slot = 1 + pass % (FX_COUNTERS - 1);
      if (pass >= FX_COUNTERS - 1) INTI_CUDA(cudaMemsetAsync(flag + slot, 0, sizeof(int), ctx->stream));
      fx_run(ctx, p, plan, w.nc, w.planes, flag + slot);
      FxOut o;
      o.rows = plan.rows;
      o.partial = ctx->fx.partial.as<double>();
      o.rowscale = plan.rowscale.as<double>();
      o.colmax = colmax;
      o.digits = fx_digits_ptr(ctx, plan, nrhs);
      o.flag = flag;
      o.rowptr = corr ? corr->rowptr.as<int64_t>() : nullptr;
      o.col = corr ? corr->col.as<int32_t>() : nullptr;
      o.val = corr ? corr->val.as<double>() : nullptr;
      o.x = x;
      o.y = y;
      o.ldx = ldx;
      o.ldy = ldy;
      o.c0 = c0;
      o.nall = nrhs;
      o.nc = w.nc;
      o.half = w.half;
      o.nslots = plan.nslots;
      o.scale = 1.0 / (4 * kPi);
      o.ar = alpha ? alpha[0] : 1.0;
      o.ai = alpha ? alpha[1] : 0.0;
      o.br = beta ? beta[0] : 0.0;
      o.bi = beta ? beta[1] : 0.0;
      o.beta_zero = o.br == 0.0 && o.bi == 0.0;
      launch_pdl(ctx->stream, dim3(plan.nrows, w.cols), FX_M, 0, &fx_finish<C>, o);
      ctx->launches++;
      if (fx_near_kind(p.kind)) {
        launch_pdl(ctx->stream, dim3((unsigned)((plan.ntargets + 31) / 32), (unsigned)((w.cols + 3) / 4)), 128, 0,
                   &fx_near_add<C>, plan.ntargets, fx_near(p, plan), x, ldx, y, ldy, c0, w.cols, o.ar, o.ai, flag);
        ctx->launches++;
      }
    }
  };
  if (cplx)
    by_type(std::true_type());
  else
    by_type(std::false_type());
  INTI_CUDA(cudaGetLastError());
}

void fx_theta(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, const double2* g0, const double2* g1, int ns,
              double2* out) {
  const bool cplx = p.pde == HELMHOLTZ;
  const int nc = fx_width(ns * (cplx ? 2 : 1));
  INTI_CUDA(cudaMemsetAsync(ctx->fx.work.p, 0, fx_work_bytes(p, plan.nsurf, ns), ctx->stream));
  int* flag = ctx->fx.work.as<int>();
  unsigned long long* colmax = fx_colmax_ptr(ctx);
  fx_theta_max<<<(unsigned)(((int64_t)plan.nstages * ns + 255) / 256), 256, 0, ctx->stream>>>(
      plan.nstages, plan.stages, ns, cplx, p.weights, g0, g1, colmax, ctx->fx.mass.as<double>());
  fx_guard_run(ctx, p, plan, ns);
  const int64_t threads = (int64_t)plan.nstages * 4 * (cplx ? nc / 2 : nc);
  auto by_type = [&](auto cc) {
    constexpr bool C = decltype(cc)::value;
    fx_theta_pack<C><<<(unsigned)((threads + 127) / 128), 128, 0, ctx->stream>>>(
        plan.nstages, plan.stages, p.weights, g0, g1, ns, nc, colmax, flag,
        ctx->fx.bdig.as<unsigned char>(), fx_digits_ptr(ctx, plan, ns));
    fx_run(ctx, p, plan, nc, 1, flag + 1);
    fx_theta_finish<C><<<dim3(plan.nrows, ns), FX_M, 0, ctx->stream>>>(
        plan.rows, ctx->fx.partial.as<double>(), plan.rowscale.as<double>(), colmax,
        fx_digits_ptr(ctx, plan, ns), ns, nc, flag, out);
    if (fx_near_kind(p.kind)) {
      const int64_t m = plan.ntargets;
      fx_near_theta<C><<<(unsigned)((m * ns + 127) / 128), 128, 0, ctx->stream>>>(m, ns, fx_near(p, plan), g0, g1, out,
                                                                                flag);
      ctx->launches++;
    }
  };
  if (cplx)
    by_type(std::true_type());
  else
    by_type(std::false_type());
  ctx->launches += 3;
  INTI_CUDA(cudaGetLastError());
}

}  // namespace inti
