// FP64 residuals and reliable updates of a block of right-hand sides (qq_pend.cu).
#pragma once
#include "qq_ctx.h"
#include "qq_mrhs.cuh"

namespace qq {

// Which right-hand sides a launch concerns: all, those awaiting their reliable update, or
// those whose residual goes back into the block.
enum PendMask : int { PEND_ALL = 0, PEND_PENDING = 1, PEND_INSERT = 2 };

struct PendArgs {
  int vh, nb;
  size_t stride;             // bytes of an FP64 field
  void* x;                   // FP64 solutions and sources: field rhs[k] belongs to
  const void* b;             //   right-hand side k of the block
  int rhs[kMaxBatch];
  void *tmp, *r64;           // FP64 scratch (odd parity) and residuals: field k
  Spinor xl, r, rhat;        // block fields
  double* S;                 // scalars, kScal per right-hand side
  unsigned* ctl;
  double tol;
  double* hist;              // true-residual history (see reliable_decide)
  int* hist_its;
  int hmax;
  double* partial;           // pend_partials doubles
};

size_t pend_partials(int vh, int nb);
// First residuals: r64 = b - A x, the scalars and the active / done masks of every
// right-hand side (S[SC_T2] = ||b||^2, S[SC_TRUE] = ||r|| / ||b||), r = rhat = r64.  ctl
// is zero before.
int pend_start(qq_ctx* c, const PendArgs& A, int prec, const double kappa[2]);
// The reliable updates of all pending right-hand sides.
int pend_update(qq_ctx* c, const PendArgs& A, int prec, const double kappa[2]);

// out[0] = ||b - (x + tk J x - kappa h)||^2, out[1] = ||b||^2 (device) on one parity's FP64
// fields.
int residual_norms(qq_ctx* c, Spinor b, Spinor x, Spinor h, double tk, double kappa, double* out);

}  // namespace qq
