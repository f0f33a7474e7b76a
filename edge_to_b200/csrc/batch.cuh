// The batched solve (batch.cu) and the one-launch 2-D V-cycle tail (vtail.cu): descriptors and launchers.
#pragma once
#include "common.cuh"
#include "element_op.cuh"

namespace edge {

constexpr int BATCH_MAXL = 8;             // levels 0..7

struct BatchLevel {
  Geo g;
  void *b, *xa, *xb, *r, *ea, *eb, *res;  // V-cycle vectors (type TV; b unused on level 0)
  const void* S;                          // stencil, levels >= 1 (type TS)
  const void* dinv;                       // Jacobi inverse diagonal (level 0: TD0, else TV)
};

// One problem of the batch: pointers into the problem's own buffers (edge_problem) and the
// solver settings of its multigrid.
struct BatchDesc {
  int n_level, nd, keep_omega, pad0;
  int sweeps[BATCH_MAXL];
  double wscale[BATCH_MAXL];  // 1.06^level
  double omega, min_omega, omega0;
  const uint8_t* mask;
  const double* E64;  // fine-level E in FP64 (the search direction's product)
  const void* ET;     // fine-level E in the V-cycle's type
  const double* K0_64;  // element matrix, corner-bit order, FP64
  const void* K0_T;     // the same in the V-cycle's type
  int wht;              // the element matrix has the box structure: k2 holds its transform
  KHat2<double> k2;
  double *b64, *x64, *r64, *p64, *q64;
  const double* Ainv;
  PcgState* st;
  const int* chol_status;
  BatchLevel lv[BATCH_MAXL];
};

// Types of a solve: FP64; or FP32 with BF16 fine Jacobi diagonals and BF16 or FP32 coarse stencils.
enum SolveKind { SOLVE_FP64, SOLVE_MIXED_BF16, SOLVE_MIXED_FP32 };

// The launchers return how many kernels they launched; an error stays in cudaGetLastError().
// Solves of the problems D[0..cnt) (order: largest first) taken from *queue (zero) by teams of `team` blocks
// (1, 2, 4, 8 or 16) of `threads` threads, on at most sm_budget SMs' worth of blocks (0: as many as
// fit); tns[2 i], tns[2 i + 1]: start and end of problem i (ns).
int batch_solve_launch(SolveKind kind, int threads, int team, const BatchDesc* D, int cnt, unsigned* queue,
                       int sm_budget, double tol, int maxiter, long long* tns, cudaStream_t stream);
// Teams of 16 blocks that the GPU holds at once (0: none).
int batch_clusters16(SolveKind kind, int threads);
// The V-cycle of one 2-D problem from its fine residual lv[0].r to the interpolated correction
// lv[0].ea, one cluster launch of VTAIL_C blocks of VTAIL_BT threads.
constexpr int VTAIL_C = 8, VTAIL_BT = 512;
int vtail2_launch(SolveKind kind, const BatchDesc& d, const double* omega_dev, cudaStream_t stream);

}  // namespace edge
