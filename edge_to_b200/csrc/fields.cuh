// Element-wise passes on arrays in the user's layout, compiled in their own translation unit
// (fields.cu).  The launchers enqueue on `stream` and return how many kernels they launched.
#pragma once
#include "common.cuh"
#include "element_op.cuh"

namespace edge {

// ------------------------------------------------------------------ OC design update
constexpr int OC_THREADS = 512;
constexpr int OC_CAND = 15;          // multipliers evaluated per pass over the elements
constexpr int OC_MAX_BLOCKS = 148;
constexpr long long OC_PART = 16LL * OC_MAX_BLOCKS;  // reduction doubles of one OC update
// Bisection state of one OC update on the device (see fields.cu) and its results.
struct OcState {
  double l1, l2, last;  // bracket, and the last multiplier tried
  double a, b;          // largest infeasible / smallest feasible multiplier known
  double change;        // sum((rho_new - rho)^2)
  int steps, done, allzero, spread;
  double lam[OC_CAND];  // candidates of the next pass
};
// rho_new = the OC update of rho with sensitivities dr; ocp: n doubles of scratch, part: OC_PART
// doubles, ticket: one counter that is zero (and left so).  The results (last, steps, change) are in
// *st and, when given, *host (pinned host memory, so that no copy is needed to read them).
int oc_launch(long long n, const double* rho, const double* dr, double A, double vol, double vf, double move,
              double* ocp, double* rho_new, double* part, unsigned* ticket, OcState* st, OcState* host,
              cudaStream_t stream);
// The OC updates of many problems in one launch: one block per problem, taken from a queue
// (*queue is zero).  lam_out, steps_out: the last multiplier and the bisection steps.
struct BatchOcDesc {
  long long n;
  const double* rho;
  const double* dr;
  double* ocp;  // n doubles of scratch
  double* rho_new;
  double A, vol, vf;
};
int oc_batch_launch(const BatchOcDesc* D, int nprob, unsigned* queue, double move, double* lam_out, int* steps_out,
                    cudaStream_t stream);

}  // namespace edge
