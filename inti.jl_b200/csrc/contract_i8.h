// Multi-column pair contractions on the INT8 tensor path (contract_i8.cu).
// Internal.
#pragma once

#include <cstdint>
#include <vector>

#include "common.h"

namespace inti {

// Kernel values of a contraction besides SL .. CF: the (S, D) pair of the
// density-interpolation Theta, and its derivative form (ADL, HS).
constexpr int FX_THETA = 6, FX_THETA_D = 7;

// A block-diagonal pair product: surface s sums its sources
// [src[s], src[s] + nsrc[s]) into its targets [row[s], row[s] + nrow[s]).
struct FxProblem {
  int pde = LAPLACE, kind = SL;
  double k = 0.0;
  double c1[2] = {1.0, 0.0}, c2[2] = {0.0, 0.0};
  const double* tcoords = nullptr;   // 3 x targets
  const double* tnormals = nullptr;  // for ADL, HS and FX_THETA_D
  const double* coords = nullptr;    // 3 x sources
  const double* normals = nullptr;
  const double* weights = nullptr;
  std::vector<int64_t> row, nrow, src, nsrc;
};

// Whether the contraction is the faster form for a product of this many targets
// and pairs (per column, summed over the surfaces).
bool fx_pays(int pde, int kind, double targets, double pairs);
// Builds the plan and sizes the buffers of a product of `ncols` columns.
// False when there is no memory for them, and while the context's stream is
// being captured: a graph would keep the addresses of buffers that the
// context replaces when a larger product needs more.
bool fx_prepare(inti_ctx* ctx, const FxProblem& p, FxPlan& plan, int ncols);
// Y = alpha*(scale*A X + C X) + beta*Y, column-major X and Y (complex
// interleaved).  A product whose densities or kernel values do not fit the
// fixed-point form (not finite, of extreme magnitude, or of magnitudes that
// differ so much within a row or column that an entry would come out worse
// than an FP64 sum) leaves Y alone and sets *fx_flag(ctx), which the caller's
// FP64 kernels then run on.
void fx_apply(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, const inti_csr* corr, const double* x,
              int64_t ldx, double* y, int64_t ldy, int nrhs, const double* alpha, const double* beta);
// Theta products S g1 - D g0 of the targets (out: m x ns complex, row-major)
// for the traces g0, g1 (sources x ns, complex); *fx_flag(ctx) as above.
void fx_theta(inti_ctx* ctx, const FxProblem& p, const FxPlan& plan, const double2* g0, const double2* g1, int ns,
              double2* out);
const int* fx_flag(const inti_ctx* ctx);
// An operator or batch takes part in (once) or leaves the users of the
// context's buffers; the last one to leave, with nothing in flight on the
// context's stream, gives them back.
void fx_hold(inti_ctx* ctx, FxPlan& plan);
void fx_drop(inti_ctx* ctx, FxPlan& plan);

}  // namespace inti
