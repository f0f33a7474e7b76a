// Many independent 2-D problems solved in one persistent launch.
//
// k_batch_pcg: a team of C blocks (one block, or a thread block cluster of C blocks) takes
// the next unsolved problem from a queue (one atomicAdd per problem; the host orders the
// problems largest first, so the long solves start first) and runs that problem's whole
// solve before taking the next: PCG with the Krylov vectors, the
// search direction's product and every inner product in FP64, preconditioned by the
// problem's V-cycle in the problem's precision (FP64; or FP32 with the BF16 fine-level Jacobi
// diagonal and BF16 coarse stencils of the mixed path), on the hierarchy that the problem's
// own set-up built (Galerkin stencils, Jacobi diagonals, the coarsest dense inverse).
//
// The V-cycle is the per-problem solver's (pre- and post-smoothing sweeps per level,
// omega * 1.06^level, full-weighting restriction and its interpolation, the exact coarsest
// solve), the PCG recurrence and the residual-driven omega schedule those of
// solvers/_multigrid_cuda.py:188-241.  Every step is one pass of the block over one level's
// nodes (the team's threads striding over them) followed by a team barrier (__syncthreads, or
// the cluster barrier with its release/acquire ordering), which makes the team's global writes
// visible to its next step (data written inside the launch is read with plain loads, never
// through the read-only path); inner products are sums in an order that does not depend on the
// team's size (TeamSum), and every other step is node by node, so a problem's result, bit for bit,
// depends neither on the team that solved it nor on the other problems (for a given block size).
// The PCG loop is bounded by maxiter; the queue counter is the only state shared between teams and
// nothing waits on it (the cluster barrier only joins the blocks of one team, which run together).
#include "batch_ops.cuh"

#include <algorithm>
#include <type_traits>

namespace edge {

// z = V-cycle(r) into lv[0].res, r the FP64 PCG residual (read in the V-cycle's type).  Levels that one block covers with
// a node per thread are smoothed by the team's first block alone: a step then ends in __syncthreads
// (1.2 us a step) instead of a cluster barrier (2.7 to 4 us on 16 blocks).  The coarsest solve, a dense
// product, is the whole team's.
template <int C, typename TV, typename TD0, typename TS>
EDGE_D void b_vcycle(const BatchDesc& d, const FineK<TV>& sK, double omega, double* sb) {
  using TM = Team<C>;
  const int L = d.n_level;
  TV* xcur[BATCH_MAXL];
  int ls = L;  // levels [ls, L): the first block's
  if constexpr (C > 1)
    while (ls > 1 && d.lv[ls - 1].g.nx * d.lv[ls - 1].g.ny <= (int)blockDim.x) --ls;
  b_down<C, TV, TD0, TS>(d, sK, omega, 0, ls, xcur);
  if (ls < L) {
    if (TM::rank() == 0) b_down<1, TV, TD0, TS>(d, sK, omega, ls, L, xcur);
    TM::sync();
  }
  b_coarse2<C, TV>(d.lv[L].g, d.Ainv, d.nd, (const TV*)d.lv[L].b, (TV*)d.lv[L].res, sb);
  TM::sync();
  if (ls < L) {
    if (TM::rank() == 0) b_up<1, TV, TD0, TS>(d, sK, omega, ls, L, xcur);
    TM::sync();
  }
  b_up<C, TV, TD0, TS>(d, sK, omega, 0, ls, xcur);
}

template <int C, typename TV, typename TD0, typename TS>
EDGE_D void b_pcg_problem(const BatchDesc& d, const FineK<TV>& sK, const double* sK64, double tol, int maxiter,
                          double* sh, double* sb) {
  using TM = Team<C>;
  const Geo& g = d.lv[0].g;
  const long long n = g.n, nv = 2 * n;
  double* x = d.x64;
  double* r = d.r64;
  double* p = d.p64;
  double* q = d.q64;
  const double* b = d.b64;
  const TV* z = (const TV*)d.lv[0].res;
  double omega = d.keep_omega ? d.st->omega : d.omega0;
  const double min_omega = d.min_omega, d_omega = d.omega - d.min_omega;
  // r = b - A x (FP64)
  b_fine2<C, double, double>(g, [&](long long s, int c) { return x[c * n + s]; }, d.E64, d.mask, sK64,
                             [&](long long s, const double* own, const double* Au) {
                               for (int c = 0; c < 2; ++c) r[c * n + s] = b[c * n + s] - Au[c];
                             });
  TM::sync();
  int ph = 0;
  const double bb = b_dot<C>(nv, b, b, sh, ph);
  int done = 0, iter = 0;
  double res = 0.0, rz = 0.0, rr = 0.0;
  if (bb == 0.0) done = 1;  // nothing to solve: residual 0, like a converged solve
  if (*d.chol_status) done = 3;
  while (!done) {
    b_vcycle<C, TV, TD0, TS>(d, sK, omega, sb);
    const double rz_new = b_dot<C>(nv, r, z, sh, ph);
    const double beta = iter == 0 ? 0.0 : rz_new / rz;
    for (long long k = TM::first(); k < nv; k += TM::stride())
      p[k] = iter == 0 ? (double)z[k] : (double)z[k] + beta * p[k];
    TM::sync();
    const double pq = TeamSum<C>::run([&](int first, int step, double& acc) {
      b_fine2<C, double, double>(g, [&](long long s, int c) { return p[c * n + s]; }, d.E64, d.mask, sK64,
                                 [&](long long s, const double* own, const double* Au) {
                                   for (int c = 0; c < 2; ++c) {
                                     q[c * n + s] = Au[c];
                                     acc += own[c] * Au[c];
                                   }
                                 }, first, step);
    }, sh, ph);
    const double alpha = rz_new / pq;
    rr = TeamSum<C>::run([&](int first, int step, double& acc) {
      for (long long k = first; k < nv; k += step) {
        x[k] = x[k] + alpha * p[k];
        const double rv = r[k] - alpha * q[k];
        r[k] = rv;
        acc += rv * rv;
      }
    }, sh, ph);
    rz = rz_new;
    ++iter;
    const double R = sqrt(rr) / sqrt(bb);
    res = R;
    if (R < tol) {
      done = 1;
    } else {
      const double Rc = fmin(fmax(R, tol), 1e-1);
      omega = min_omega + d_omega / 2.0 * exp((-Rc + tol) * 500.0);
      if (iter >= maxiter) done = 2;
    }
  }
  if (TM::first() == 0) {
    PcgState* st = d.st;
    st->bb = bb;
    st->rr = rr;
    st->rz = rz;
    st->res = res;
    st->iter = iter;
    st->done = done;
    st->omega = omega;
  }
}

// The batched solve.  C > 1: launched as thread block clusters of C blocks (cluster
// dimension set at launch); rank 0 of a team takes the team's problems from the queue.
EDGE_D long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// tns (may be null): start and end of each problem's solve (global timer, ns), for the
// benchmark's load-balance record.
//
// The 1,024-thread forms sit at the limit of 64 registers and spill (teams of 4, bytes stored / loaded:
// mixed 1,992 / 3,188, FP64 5,168 / 8,060); the 512-thread forms have 128 and spill 12 to 40 bytes.
template <typename TV, typename TD0, typename TS, int BT, int C>
__global__ void __launch_bounds__(BT) k_batch_pcg(const BatchDesc* D, int nprob, unsigned* queue, double tol,
                                                  int maxiter, long long* tns) {
  using TM = Team<C>;
  __shared__ double sh[TeamSum<C>::SH];
  __shared__ double sb[BATCH_COARSE_SMEM];
  __shared__ TV sK[64];
  __shared__ double sK64[64];
  __shared__ KHat2<TV> sk2;
  __shared__ BatchDesc sd;
  __shared__ int s_idx;
  for (;;) {
    if (TM::first() == 0) s_idx = (int)atomicAdd(queue, 1u);
    TM::sync();
    int idx;
    if constexpr (C == 1) idx = s_idx;
    else idx = *cooperative_groups::this_cluster().map_shared_rank(&s_idx, 0);
    TM::sync();  // every block has read rank 0's s_idx before rank 0 may exit or overwrite it
    if (idx >= nprob) return;
    {
      const int* src = reinterpret_cast<const int*>(D + idx);
      int* dst = reinterpret_cast<int*>(&sd);
      for (int k = threadIdx.x; k < (int)(sizeof(BatchDesc) / sizeof(int)); k += BT) dst[k] = src[k];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 64; k += BT) {
      sK[k] = reinterpret_cast<const TV*>(sd.K0_T)[k];
      sK64[k] = sd.K0_64[k];
    }
    if (threadIdx.x < 24) {
      const double* src = &sd.k2.dg[0][0];
      reinterpret_cast<TV*>(&sk2)[threadIdx.x] = (TV)src[threadIdx.x];
    }
    __syncthreads();
    const FineK<TV> fk{sK, sd.wht ? &sk2 : nullptr};
    const long long t0 = global_ns();
    b_pcg_problem<C, TV, TD0, TS>(sd, fk, sK64, tol, maxiter, sh, sb);
    TM::sync();
    if (tns && TM::first() == 0) {
      tns[2 * idx] = t0;
      tns[2 * idx + 1] = global_ns();
    }
  }
}

// One persistent launch.
template <typename TV, typename TD0, typename TS, int BT, int C>
static int batch_go(const BatchDesc* D, int cnt, unsigned* queue, int sm_budget, double tol, int maxiter,
                    long long* tns, cudaStream_t stream) {
  auto kern = k_batch_pcg<TV, TD0, TS, BT, C>;
  if constexpr (C > 8) cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int budget = sm_budget > 0 ? std::min(sm_budget, sms) : sms;
  if constexpr (C == 1) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BT, 0);
    const int grid = std::max(1, std::min(cnt, std::max(1, per_sm) * budget));
    kern<<<grid, BT, 0, stream>>>(D, cnt, queue, tol, maxiter, tns);
  } else {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C * sms);
    cfg.blockDim = dim3(BT);
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg);
    const int fit = std::max(1, clusters * budget / sms);
    const int teams = std::max(1, std::min(cnt, fit));
    cfg.gridDim = dim3(C * teams);
    cudaLaunchKernelEx(&cfg, kern, D, cnt, queue, tol, maxiter, tns);
  }
  return 1;
}
template <typename TV, typename TD0, typename TS, int BT> static int clusters16() {
  auto kern = k_batch_pcg<TV, TD0, TS, BT, 16>;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 16;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(BT);
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return clusters;
}
template <typename TV, typename TD0, typename TS>
static int batch_kind(int threads, int team, const BatchDesc* D, int cnt, unsigned* queue, int sm_budget, double tol,
                      int maxiter, long long* tns, cudaStream_t st) {
  auto go = [&](auto bt) {
    constexpr int BT = decltype(bt)::value;
    switch (team) {
      case 2: return batch_go<TV, TD0, TS, BT, 2>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
      case 4: return batch_go<TV, TD0, TS, BT, 4>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
      case 8: return batch_go<TV, TD0, TS, BT, 8>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
      case 16: return batch_go<TV, TD0, TS, BT, 16>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
      default: return batch_go<TV, TD0, TS, BT, 1>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
    }
  };
  if (threads == 1024) return go(std::integral_constant<int, 1024>{});
  if (threads == 256 && team == 1)
    return batch_go<TV, TD0, TS, 256, 1>(D, cnt, queue, sm_budget, tol, maxiter, tns, st);
  return go(std::integral_constant<int, 512>{});
}
int batch_solve_launch(SolveKind kind, int threads, int team, const BatchDesc* D, int cnt, unsigned* queue,
                       int sm_budget, double tol, int maxiter, long long* tns, cudaStream_t st) {
  using bf = __nv_bfloat16;
  switch (kind) {
    case SOLVE_FP64:
      return batch_kind<double, double, double>(threads, team, D, cnt, queue, sm_budget, tol, maxiter, tns, st);
    case SOLVE_MIXED_BF16:
      return batch_kind<float, bf, bf>(threads, team, D, cnt, queue, sm_budget, tol, maxiter, tns, st);
    default: return batch_kind<float, bf, float>(threads, team, D, cnt, queue, sm_budget, tol, maxiter, tns, st);
  }
}
int batch_clusters16(SolveKind kind, int threads) {
  using bf = __nv_bfloat16;
  const bool big = threads == 1024;
  switch (kind) {
    case SOLVE_FP64: return big ? clusters16<double, double, double, 1024>() : clusters16<double, double, double, 512>();
    case SOLVE_MIXED_BF16: return big ? clusters16<float, bf, bf, 1024>() : clusters16<float, bf, bf, 512>();
    default: return big ? clusters16<float, bf, float, 1024>() : clusters16<float, bf, float, 512>();
  }
}

}  // namespace edge
