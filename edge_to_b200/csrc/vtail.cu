// The one-launch 2-D V-cycle below the fine level (declared in batch.cuh).  A translation unit of its own:
// a process loads a unit's kernels at its first launch from it, and together with the batched solve's 33
// kernels that made the first 2-D solve of a process 68 ms instead of 11.
#include "batch_ops.cuh"

namespace edge {

// The V-cycle of one 2-D problem below its fine level as one launch of a thread block cluster, for the
// per-problem solver: restriction of the fine residual, all coarse levels, the coarsest solve and the
// interpolation back to the fine level (lv[0].r -> lv[0].ea), with the passes above.  As separate
// launches each step costs 3.5 us of which the pass itself is a fraction (nine launches per level with
// three sweeps); here a step ends in a cluster barrier or, on the levels one block covers, in
// __syncthreads.
template <typename TV, typename TS, int BT, int C>
__global__ void __launch_bounds__(BT) k_vtail2(const __grid_constant__ BatchDesc d, const double* omega_dev) {
  EDGE_PDL_ENTRY();
  using TM = Team<C>;
  __shared__ double sb[BATCH_COARSE_SMEM];
  const double omega = *(const volatile double*)omega_dev;
  const int L = d.n_level;
  TV* xcur[BATCH_MAXL];
  const FineK<TV> none{nullptr, nullptr};
  const bool j0 = L > 1 && d.sweeps[1] >= 1;
  b_restrict2<C, TV>(d.lv[0].g, d.lv[1].g, (const TV*)d.lv[0].r, (TV*)d.lv[1].b, (const TV*)d.lv[1].dinv,
                     Conv<TV>::from(omega * d.wscale[1]), j0 ? (TV*)d.lv[1].xa : nullptr);
  TM::sync();
  int ls = L;  // levels [ls, L): the first block's
  while (ls > 1 && d.lv[ls - 1].g.nx * d.lv[ls - 1].g.ny <= BT) --ls;
  b_down<C, TV, TV, TS>(d, none, omega, 1, ls, xcur);
  if (ls < L) {
    if (TM::rank() == 0) b_down<1, TV, TV, TS>(d, none, omega, ls, L, xcur);
    TM::sync();
  }
  b_coarse2<C, TV>(d.lv[L].g, d.Ainv, d.nd, (const TV*)d.lv[L].b, (TV*)d.lv[L].res, sb);
  TM::sync();
  if (ls < L) {
    if (TM::rank() == 0) b_up<1, TV, TV, TS>(d, none, omega, ls, L, xcur);
    TM::sync();
  }
  b_up<C, TV, TV, TS>(d, none, omega, 1, ls, xcur);
  b_prolong2<C, TV>(d.lv[0].g, d.lv[1].g, (const TV*)d.lv[1].res, (TV*)d.lv[0].ea);
}

int vtail2_launch(SolveKind kind, const BatchDesc& d, const double* omega_dev, cudaStream_t stream) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = VTAIL_C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(VTAIL_C);
  cfg.blockDim = dim3(VTAIL_BT);
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  switch (kind) {
    case SOLVE_FP64: cudaLaunchKernelEx(&cfg, k_vtail2<double, double, VTAIL_BT, VTAIL_C>, d, omega_dev); break;
    case SOLVE_MIXED_BF16: cudaLaunchKernelEx(&cfg, k_vtail2<float, __nv_bfloat16, VTAIL_BT, VTAIL_C>, d, omega_dev); break;
    default: cudaLaunchKernelEx(&cfg, k_vtail2<float, float, VTAIL_BT, VTAIL_C>, d, omega_dev); break;
  }
  return 1;
}

}  // namespace edge
