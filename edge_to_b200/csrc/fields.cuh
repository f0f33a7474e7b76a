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

// ------------------------------------------------------------------ density filter
// Cone filter (geom/_filters.py:72-161, core/_filter.py:78-124): taps o_k with global weights w_k;
// (H rho)_e = sum_k w_k rho_{e+o_k} / N_e with N_e = sum of the in-bounds w_k.
constexpr int MAX_TAPS = 128;
struct Taps {
  int n;
  int off[MAX_TAPS][3];  // (dx, dy, dz) in element units
  double w[MAX_TAPS];
};
// The taps by columns along the middle element axis (y in 3-D, x in 2-D) for the tiled kernels:
// column c is at offset (o0, o2) of the slowest and fastest axis and holds the weights of the
// middle offsets -R..R (present: bit b for offset b - R).
constexpr int FT_RMAX = 3;
constexpr int FT_COLS = (2 * FT_RMAX + 1) * (2 * FT_RMAX + 1);
struct TapCols {
  int n, R, R0;  // columns; tile halo along the middle and fastest axes, along the slowest
  double nint;   // N_e of an element whose taps are all in bounds
  signed char o0[FT_COLS], o2[FT_COLS];
  unsigned char present[FT_COLS];
  double w[FT_COLS][2 * FT_RMAX + 1];
};
// false when a tap repeats or reaches further than FT_RMAX: the one-thread-per-element kernels
bool make_tap_cols(int dim, const Taps& t, TapCols& c);
// What the forward filter stores: H rho, and for the SIMP law (MaterialModels.py:47-60) the
// penalised density clip((H rho)^p, void, 1) at the element's slot of `slots`.
struct FilterOut {
  double* rho_f;
  double* E64;  // null: no law
  float* E32;   // may be null
  double penalty, vmin;
  Geo slots;    // node grid of the element slots (rows may be longer than the filter's grid)
};
int filter_forward(const Geo& g, const Taps& t, const TapCols* c, const double* N, const double* in,
                   const FilterOut& out, cudaStream_t stream);
int filter_transpose(const Geo& g, const Taps& t, const TapCols* c, const double* N, const double* in, double* out,
                     cudaStream_t stream);
int filter_norm(const Geo& g, const Taps& t, double* N, cudaStream_t stream);

// ------------------------------------------------------------------ operator on user vectors
// Element matrix of a 2-D problem, corner-bit order, row-major.
struct K2Dense {
  double k[64];
};
// out = K(E) u with identity rows on constrained DOFs, u and out in the user's layout
// (v[2 node + c], node = j nx + i); E and mask in the slots of g.
int product2_user(const Geo& g, const K2Dense& K, const double* E, const uint8_t* mask, const double* u, double* out,
                  cudaStream_t stream);
// dk_e = -u_e^T K0 u_e per element (reference element order) from a user-layout displacement; box: the
// transformed element matrix when it has the box structure, else null
int energy2_user(const Geo& g, const K2Dense& K, const KHat2<double>* box, const double* u, double* dk,
                 cudaStream_t stream);

// The same in 3-D, for element matrices with the box structure (KHat3, element_op.cuh) and, when
// `cube` is given, its block form (equal edges, isotropic material: KCube64).  ly: user3_rows of the grid.
struct KCube64 {
  double nd, no, sh, bd, bo, td, to, h7;  // nd and td without the shared part no / to
};
int product3_user(const Geo& g, const KHat3<double>& K, const KCube64* cube, const double* E, const uint8_t* mask,
                  const uint8_t* eflag16, int mpz, int ly, const double* u, double* out, cudaStream_t stream);
int energy3_user(const Geo& g, const KHat3<double>& K, const KCube64* cube, int ly, const double* u, double* dk,
                 cudaStream_t stream);
int user3_rows(const Geo& g, bool product);
// Grids that the products (or energies) above take: their tile counts are grid dimensions.
bool user_grid_ok(const Geo& g, bool product);

// ------------------------------------------------------------------ coarsest level
// Inverse of a symmetric positive definite matrix.  A: np x np row-major, np = inv_padded(nd), the nd x nd
// matrix in its upper left corner and zeros elsewhere (overwritten); Ainv: nd x nd; work: inv_work(nd)
// doubles.  *status is set to 1 on a pivot that is not positive (taken as 1 then).
constexpr int INV_B = 64;
inline int inv_padded(int nd) { return (nd + INV_B - 1) / INV_B * INV_B; }
inline long long inv_work(int nd) { return 2LL * INV_B * inv_padded(nd) + 2LL * INV_B * INV_B; }
int spd_inverse(double* A, int nd, double* Ainv, double* work, int* status, cudaStream_t stream);

}  // namespace edge
