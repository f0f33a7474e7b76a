// Element-wise passes on arrays in the user's layout (declared in fields.cuh).
#include "fields.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

namespace edge {

// ------------------------------------------------------------------ OC design update
// The OC update of TopOpt/_cuda.py:242-280: ocP = max(1e-12, rho sqrt(max(-dr / A, 0))) (1e-3
// everywhere when all are zero, MaterialModels.py:75-88), the bisection of the multiplier in
// [1e-9, 1e9] until (l2 - l1) / (l2 + l1) <= 1e-4 (at most 200 steps), rho_new at the last
// multiplier tried and sum((rho_new - rho)^2).
//
// What bounds it: the bisection is a serial chain of about 45 decisions "is sum(rho_new(mid)) A
// <= vf vol", each a sum over all elements.  The sum does not increase with the multiplier, so a
// decision is known without a sum when mid lies outside the interval (a, b) between the
// largest multiplier seen to be infeasible and the smallest seen to be feasible.  A pass
// therefore evaluates OC_CAND multipliers spread evenly in log over (a, b), which takes the
// 16th root of its ratio: four passes from 1e18 to 1.0007; then the few midpoints that still
// fall inside (a, b) are evaluated as a tree, four deep per pass, and walked exactly as the
// sequential bisection would, so the multiplier used is a midpoint of that bisection, decided
// on an evaluated sum or by monotonicity.  A pass ends in the block that finishes last: it sums
// the blocks' partials, moves the bracket and leaves the next candidates; no block waits for
// another.  The number of passes is fixed (OC_PASSES), those after the end return at once, so
// neither a host read nor a graph condition is needed between them.
//
// A candidate costs one multiply by the reciprocal multiplier, the two bounds and one FMA per
// element (rho_new itself is divided, as the reference does).
constexpr int OC_PASSES = 6;  // four spread, one of the tree, one more when the first only finds all ocP zero

// The upper ends of the bracket while every midpoint is feasible: l2[k + 1] = (1e-9 + l2[k]) / 2,
// all of them far from the end of the bisection (the bracket stays wider than 4 to 1).  Most
// updates begin with about 30 such steps; a chain of dependent FP64 operations, walked here by
// bisection on the step number instead.
constexpr int OC_CHAIN = 57;
struct OcChain {
  double l2[OC_CHAIN + 1];
};
constexpr OcChain make_oc_chain() {
  OcChain c{};
  c.l2[0] = 1e9;
  for (int k = 0; k < OC_CHAIN; ++k) c.l2[k + 1] = 0.5 * (1e-9 + c.l2[k]);
  return c;
}
__constant__ OcChain c_oc_chain = make_oc_chain();
static_assert(make_oc_chain().l2[OC_CHAIN] > 4e-9, "the chain ends before the bracket closes");

// Bisection bracket; mids outside (a, b) are decided by monotonicity.
struct OcBis {
  double l1, l2, last, a, b;
  int steps;
  // (l2 - l1) / (l2 + l1) > 1e-4; the division only where rounding could decide it
  EDGE_D bool open() const {
    const double d = l2 - l1, s = l2 + l1;
    bool o = d > 1.0000001e-4 * s;
    if (!o && d > 0.9999999e-4 * s) o = d / s > 1e-4;
    return o && steps < 200;
  }
  EDGE_D void take(bool valid) {
    const double mid = 0.5 * (l1 + l2);
    if (valid) l2 = mid;
    else l1 = mid;
    last = mid;
    ++steps;
  }
  // decides midpoints while they lie outside (a, b); true: the bisection has ended
  EDGE_D bool advance() {
    if (steps < OC_CHAIN && l1 == 1e-9 && l2 == c_oc_chain.l2[steps]) {
      // every step so far was feasible: the last k with c_oc_chain.l2[k] >= b, by halving
      int k = steps;
#pragma unroll
      for (int h = 32; h >= 1; h >>= 1)
        if (k + h <= OC_CHAIN && c_oc_chain.l2[k + h] >= b) k += h;
      if (k > steps) {
        last = l2 = c_oc_chain.l2[k];
        steps = k;
      }
    }
    while (open()) {
      const double mid = 0.5 * (l1 + l2);
      if (mid >= b) take(true);
      else if (mid <= a) take(false);
      else return false;
    }
    return true;
  }
  EDGE_D void decide(bool valid) {  // outcome of an evaluated midpoint
    const double mid = 0.5 * (l1 + l2);
    if (valid) b = mid;
    else a = mid;
    take(valid);
  }
};

// Sum of v[0..15] over the block's threads into out[0..15] (shared memory, valid after the
// block's next barrier); sw: 16 doubles per warp of scratch.  A warp folds the 16 values across
// its lanes (each exchange halves the values a lane still carries): 16 exchanges for 16 sums.
EDGE_D void block_sum16(double v[16], double* sw, double* out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int h = 8; h >= 1; h >>= 1) {
    const bool up = lane & h;
#pragma unroll
    for (int t = 0; t < 8; ++t)
      if (t < h) {
        const double keep = up ? v[t + h] : v[t], give = up ? v[t] : v[t + h];
        v[t] = keep + __shfl_xor_sync(0xffffffffu, give, h);
      }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
  if (lane < 16) sw[wid * 16 + lane] = v[0];  // lane t of every warp holds the warp's sum of value t
  __syncthreads();
  if (wid < 16) {  // warp t finishes value t (at least 16 warps)
    double s = lane < nw ? sw[lane * 16 + wid] : 0.0;
    s = warp_sum(s);
    if (lane == 0) out[wid] = s;
  }
}

// Where a pass evaluates need not be exact, only ascending inside (ca, cb): FP32 logarithm and
// power (the ratio is at least 1.002, its 16th root 1000 FP32 roundings above 1).
EDGE_D double oc_spread(double ca, double cb, int t) {
  const float l = log2f(__fdividef((float)cb, (float)ca));
  const double lam = ca * (double)exp2f(l * ((t + 1) * 0.0625f));
  return lam < cb ? lam : cb;
}
EDGE_D double oc_value(double r, double o, double lam, double move) {
  const double xU = fmin(fmax(r + move, 0.0), 1.0);
  const double xL = fmin(fmax(r - move, 0.0), 1.0);
  return fmax(0.0, fmax(xL, fmin(1.0, fmin(xU, o / lam))));
}

// The interval of multipliers not yet known to be feasible or infeasible is wide: spread.
EDGE_D bool oc_wide(const OcBis& B) { return B.b > 1.002 * B.a; }
// sum / vol <= vf; the division only where rounding could decide it.
EDGE_D bool oc_feasible(double sum, double vol, double vf) {
  const double t = vf * vol;
  if (vol > 0.0 && sum < t * 0.999999999) return true;
  if (vol > 0.0 && sum > t * 1.000000001 && t > 0.0) return false;
  return sum / vol <= vf;
}
// Moves the bracket by the outcomes of one pass (bit t of ok: candidate t is feasible); true: the
// bisection has ended.  The bisection itself only starts once (a, b) is narrow.
EDGE_D bool oc_move(OcBis& B, bool spread, unsigned ok, const double* lam) {
  if (spread) {
    // the candidates ascend: the first feasible one bounds (a, b) above, the one before it below
    const int t = __ffs(ok) - 1;
    if (t >= 0) B.b = lam[t];
    if (t != 0) B.a = lam[(t > 0 ? t : OC_CAND) - 1];
    return oc_wide(B) ? false : B.advance();
  }
  bool done = false;
  int t = 0;
  for (int d = 0; d < 4 && !done; ++d) {
    const bool valid = (ok >> t) & 1;
    B.decide(valid);
    done = B.advance();
    t = 2 * t + (valid ? 1 : 2);
  }
  return done;
}
// Candidate t of the pass after bracket B: spread over (a, b) while that is wide, then the
// heap-ordered tree of undecided midpoints (the bits of the node give the outcomes on its path).
EDGE_D double oc_candidate(OcBis C, int t) {
  if (oc_wide(C)) return oc_spread(C.a, C.b, t);
  const int node = t + 1;
  bool end = false;
  for (int d = 30 - __clz(node); d >= 0 && !end; --d) {
    C.decide(!((node >> d) & 1));  // left child: feasible
    end = C.advance();
  }
  return 0.5 * (C.l1 + C.l2);
}
// (a, b) starts at the bracket's ends: every midpoint lies strictly between them
EDGE_D OcBis oc_start() { return OcBis{1e-9, 1e9, 0.5 * (1e-9 + 1e9), 1e-9, 1e9, 0}; }
EDGE_D double oc_raw(double r, double dr, double A) {
  const double o = r * sqrt(fmax(-dr / A, 0.0));
  return isnan(o) ? 0.0 : o;
}
// The candidates' design values of one element (move limits xl, xu; o not NaN: at least 1e-12)
// times A, added to v.
EDGE_D double oc_clip01(double x) {  // fmin(fmax(x, 0), 1): 0 for a NaN
  x = x > 0.0 ? x : 0.0;
  return x < 1.0 ? x : 1.0;
}
EDGE_D void oc_eval(double r, double o, double move, double A, const double* ilam, double v[16]) {
  const double xu = oc_clip01(r + move), xl = oc_clip01(r - move);
#pragma unroll
  for (int t = 0; t < OC_CAND; ++t) {
    double x = o * ilam[t];
    x = x < xu ? x : xu;
    x = x > xl ? x : xl;
    v[t] = fma(x, A, v[t]);
  }
}

// One pass.  PASS 0 computes ocP as well; PASS 2 (the third pass and later) is launched so that its
// blocks may start while the pass before is still finishing: rho and ocP are settled by then
// (the pass before let its dependents start after pass 0 had completed), so each thread fetches
// its first elements before it waits for that pass's candidates.
template <int PASS>
__global__ void __launch_bounds__(OC_THREADS)
k_oc_bisect(long long n, const double* __restrict__ rho, const double* __restrict__ dr, double A, double vol, double vf,
            double move, double* __restrict__ ocp, double* part, unsigned* ticket, OcState* st) {
  constexpr int PRE = 2;
  __shared__ double sw[16 * 16];
  __shared__ double ssum[16];
  __shared__ double slam[16], silam[16];
  __shared__ bool am_last;
  __shared__ OcBis sB;
  const long long i0 = blockIdx.x * (long long)OC_THREADS + threadIdx.x, T = (long long)gridDim.x * OC_THREADS;
  double pr[PRE], po[PRE];
  if constexpr (PASS == 2) {
#pragma unroll
    for (int q = 0; q < PRE; ++q) {
      const long long i = i0 + q * T < n ? i0 + q * T : n - 1;
      pr[q] = rho[i];
      po[q] = ocp[i];
    }
  }
  EDGE_PDL_ENTRY();
  if (PASS != 0 && st->done) return;
  const bool allz = PASS == 0 ? false : st->allzero != 0;
  if (threadIdx.x < OC_CAND) {
    const double lam = PASS == 0 ? oc_spread(1e-9, 1e9, threadIdx.x) : st->lam[threadIdx.x];
    slam[threadIdx.x] = lam;
    silam[threadIdx.x] = 1.0 / lam;
  }
  __syncthreads();
  double v[16];
#pragma unroll
  for (int t = 0; t < 16; ++t) v[t] = 0.0;
  bool any = false;
  long long i = i0;
  if constexpr (PASS == 2) {
#pragma unroll
    for (int q = 0; q < PRE; ++q)
      if (i0 + q * T < n) oc_eval(pr[q], allz ? 1e-3 : po[q], move, A, silam, v);
    i += PRE * T;
  }
  constexpr int U = 4;  // elements fetched together
  for (; i < n; i += U * T) {
    double r[U], o[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const long long iq = i + q * T < n ? i + q * T : n - 1;
      r[q] = rho[iq];
      o[q] = PASS == 0 ? dr[iq] : ocp[iq];
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (i + q * T >= n) break;
      if constexpr (PASS == 0) {
        o[q] = oc_raw(r[q], o[q], A);
        any = any || o[q] != 0.0;
        o[q] = fmax(1e-12, o[q]);
        ocp[i + q * T] = o[q];
      }
      oc_eval(r[q], allz ? 1e-3 : o[q], move, A, silam, v);
    }
  }
  v[15] = any ? 1.0 : 0.0;
  block_sum16(v, sw, ssum);
  __syncthreads();
  if (threadIdx.x < 16) {
    part[threadIdx.x * OC_MAX_BLOCKS + blockIdx.x] = ssum[threadIdx.x];
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) am_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;  // 16 warps, one per value
  double s = 0.0;
  for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(part + wid * OC_MAX_BLOCKS + b);
  s = warp_sum(s);
  if (lane == 0) ssum[wid] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    const unsigned ok = __ballot_sync(0xffffffffu, lane < OC_CAND && oc_feasible(ssum[lane & 15], vol, vf));
    if (lane == 0) {
      *ticket = 0u;
      OcBis B = oc_start();
      bool done = false;
      if constexpr (PASS == 0) {
        const bool some = ssum[15] != 0.0;  // no sensitivities: the passes that follow evaluate the fallback
        st->allzero = some ? 0 : 1;
        if (some) done = oc_move(B, true, ok, slam);
      } else {
        B = OcBis{st->l1, st->l2, st->last, st->a, st->b, st->steps};
        done = oc_move(B, st->spread != 0, ok, slam);
      }
      st->l1 = B.l1;
      st->l2 = B.l2;
      st->last = B.last;
      st->a = B.a;
      st->b = B.b;
      st->steps = B.steps;
      st->done = done ? 1 : 0;
      st->spread = oc_wide(B) ? 1 : 0;
      sB = B;
    }
    __syncwarp();
    if (lane < OC_CAND) st->lam[lane] = oc_candidate(sB, lane);
  }
}

__global__ void __launch_bounds__(OC_THREADS)
k_oc_design(long long n, const double* __restrict__ rho, const double* __restrict__ ocp, double move,
            double* __restrict__ rho_new, double* part, unsigned* ticket, OcState* st, OcState* host) {
  EDGE_PDL_ENTRY();
  const double lam = st->last;
  const bool allz = st->allzero != 0;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)OC_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * OC_THREADS) {
    const double r = rho[i];
    const double x = oc_value(r, allz ? 1e-3 : ocp[i], lam, move);
    rho_new[i] = x;
    acc += (x - r) * (x - r);
  }
  __shared__ double sh[32];
  const double bt = block_sum(acc, sh);
  grid_reduce_finish(bt, part, ticket, [=](double t) {
    st->change = t;
    if (host) {
      host->last = lam;
      host->steps = st->steps;
      host->change = t;
    }
  });
}

// The passes of k_oc_bisect by one thread block cluster of C blocks (C = 1: one block), for
// element counts that leave most of the grid's passes waiting: the whole update is one launch,
// a pass ends in a cluster barrier (the block sums go to every block's shared memory, which then
// moves the bracket and forms the next candidates by itself) instead of a launch boundary.
template <int C, int BT>
EDGE_D void oc_team(const BatchOcDesc& d, double move, double& last, int& steps, double& change) {
  constexpr int REG = 8;  // elements a thread keeps in registers
  namespace cg = cooperative_groups;
  __shared__ double sw[(BT / 32) * 16];
  __shared__ double ssum[16], slam[16], silam[16];
  __shared__ double sall[2][C][16];
  __shared__ OcBis sB;
  __shared__ int s_done, s_allz;
  unsigned rank = 0;
  if constexpr (C > 1) {
    rank = cg::this_cluster().block_rank();
    // a peer's shared memory may be written once that block has started: arrive here, wait below, so
    // that the elements' loads hide the barrier
    cg::this_cluster().barrier_arrive();
  }
  const long long i0 = rank * (long long)BT + threadIdx.x, T = (long long)C * BT;
  double rr[REG], oo[REG];
  bool any = false;
#pragma unroll
  for (int q = 0; q < REG; ++q) {
    const long long i = i0 + q * T;
    rr[q] = oo[q] = 0.0;
    if (i < d.n) {
      rr[q] = d.rho[i];
      const double o = oc_raw(rr[q], d.dr[i], d.A);
      any = any || o != 0.0;
      oo[q] = fmax(1e-12, o);
    }
  }
  for (long long i = i0 + REG * T; i < d.n; i += T) {
    const double o = oc_raw(d.rho[i], d.dr[i], d.A);
    any = any || o != 0.0;
    d.ocp[i] = fmax(1e-12, o);
  }
  if constexpr (C > 1) cg::this_cluster().barrier_wait();
  int buf = 0;
  // team sums of v[0..15] -> ssum (the same in every block)
  auto team_sum = [&](double v[16]) {
    block_sum16(v, sw, ssum);
    __syncthreads();
    if constexpr (C > 1) {
      auto cl = cg::this_cluster();
      for (int k = threadIdx.x; k < 16 * C; k += BT) *cl.map_shared_rank(&sall[buf][rank][k & 15], k >> 4) = ssum[k & 15];
      cl.sync();
      if (threadIdx.x < 16) {
        double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < C; ++k) s4[k & 3] += sall[buf][k][threadIdx.x];
        ssum[threadIdx.x] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      }
      buf ^= 1;  // this buffer is written again two sums from now, behind the next sum's barrier
      __syncthreads();
    }
  };
  if (threadIdx.x == 0) {
    sB = oc_start();
    s_done = 0;
    s_allz = 0;
  }
  __syncthreads();
  for (int pass = 0; pass < 200 && !s_done; ++pass) {
    if (threadIdx.x < OC_CAND) {
      const double lam = oc_candidate(sB, threadIdx.x);
      slam[threadIdx.x] = lam;
      silam[threadIdx.x] = 1.0 / lam;
    }
    __syncthreads();
    const bool allz = s_allz != 0;
    double v[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) v[t] = 0.0;
#pragma unroll
    for (int q = 0; q < REG; ++q)
      if (i0 + q * T < d.n) oc_eval(rr[q], allz ? 1e-3 : oo[q], move, d.A, silam, v);
    for (long long i = i0 + REG * T; i < d.n; i += T) oc_eval(d.rho[i], allz ? 1e-3 : d.ocp[i], move, d.A, silam, v);
    v[15] = any ? 1.0 : 0.0;
    team_sum(v);
    if (threadIdx.x < 32) {
      const unsigned ok = __ballot_sync(0xffffffffu, threadIdx.x < OC_CAND && oc_feasible(ssum[threadIdx.x & 15], d.vol, d.vf));
      if (threadIdx.x == 0) {
        OcBis B = sB;
        if (pass == 0 && ssum[15] == 0.0)
          s_allz = 1;  // no sensitivities: the passes that follow evaluate the fallback
        else
          s_done = oc_move(B, oc_wide(B), ok, slam) ? 1 : 0;
        sB = B;
      }
    }
    __syncthreads();
  }
  last = sB.last;
  steps = sB.steps;
  const bool allz = s_allz != 0;
  double v[16];
#pragma unroll
  for (int t = 0; t < 16; ++t) v[t] = 0.0;
#pragma unroll
  for (int q = 0; q < REG; ++q) {
    const long long i = i0 + q * T;
    if (i < d.n) {
      const double x = oc_value(rr[q], allz ? 1e-3 : oo[q], last, move);
      d.rho_new[i] = x;
      v[0] += (x - rr[q]) * (x - rr[q]);
    }
  }
  for (long long i = i0 + REG * T; i < d.n; i += T) {
    const double r = d.rho[i], x = oc_value(r, allz ? 1e-3 : d.ocp[i], last, move);
    d.rho_new[i] = x;
    v[0] += (x - r) * (x - r);
  }
  team_sum(v);  // every block has read its shared memory's remote writes when this returns
  change = ssum[0];
  __syncthreads();
}

constexpr int OC_TEAM = 16, OC_TEAM_THREADS = 512;
__global__ void __launch_bounds__(OC_TEAM_THREADS)
k_oc_cluster(BatchOcDesc d, double move, OcState* st, OcState* host) {
  EDGE_PDL_ENTRY();
  double last, change;
  int steps;
  oc_team<OC_TEAM, OC_TEAM_THREADS>(d, move, last, steps, change);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->last = last;
    st->steps = steps;
    st->change = change;
    if (host) {
      host->last = last;
      host->steps = steps;
      host->change = change;
    }
  }
}

// One block per problem, taken from a queue.
constexpr int OCB_THREADS = 512;
__global__ void __launch_bounds__(OCB_THREADS)
k_oc_batch(const BatchOcDesc* D, int nprob, unsigned* queue, double move, double* lam_out, int* steps_out) {
  __shared__ int s_idx;
  for (;;) {
    if (threadIdx.x == 0) s_idx = (int)atomicAdd(queue, 1u);
    __syncthreads();
    const int idx = s_idx;
    __syncthreads();
    if (idx >= nprob) return;
    double last, change;
    int steps;
    oc_team<1, OCB_THREADS>(D[idx], move, last, steps, change);
    if (threadIdx.x == 0) {
      lam_out[idx] = last;
      steps_out[idx] = steps;
    }
    __syncthreads();
  }
}

// One cluster up to OC_CLUSTER_MAX elements, the whole grid beyond.  A call (with its host read) in
// us, cluster / grid: 4,800 elements 40 / 57, 20,000 45 / 58, 49,152 53 / 62, 65,536 59 / 59, 110,592
// 82 / 61, 221,184 129 / 67: the cluster's 16 SMs run out of FP64 rate (four operations per element and
// candidate), the grid's passes cost their launches whatever the size.  The launches with host
// reads and divisions that both replace took 356 us at 4,800, 363 at 65,536, 776 at 524,288
// (now 83) and 2,086 at 4.2M elements (now 295).
constexpr long long OC_CLUSTER_MAX = 49152;

int oc_launch(long long n, const double* rho, const double* dr, double A, double vol, double vf, double move,
              double* ocp, double* rho_new, double* part, unsigned* ticket, OcState* st, OcState* host,
              cudaStream_t stream) {
  cudaLaunchAttribute at[1];
  cudaLaunchConfig_t cfg = {};
  cfg.stream = stream;
  cfg.attrs = at;
  if (n <= OC_CLUSTER_MAX) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = OC_TEAM;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(OC_TEAM);
    cfg.blockDim = dim3(OC_TEAM_THREADS);
    // the attribute on every call: it belongs to the current device's context, not to the process
    if (cudaFuncSetAttribute(k_oc_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaLaunchKernelEx(&cfg, k_oc_cluster, BatchOcDesc{n, rho, dr, ocp, rho_new, A, vol, vf}, move, st, host) ==
            cudaSuccess)
      return 1;
    cudaGetLastError();  // 16 blocks do not fit side by side (a part of a GPU): the grid's passes take any size
  }
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)std::min<long long>((n + OC_THREADS - 1) / OC_THREADS, OC_MAX_BLOCKS));
  cfg.blockDim = dim3(OC_THREADS);
  cfg.numAttrs = 0;  // the first pass follows whatever produced its inputs
  cudaLaunchKernelEx(&cfg, k_oc_bisect<0>, n, rho, dr, A, vol, vf, move, ocp, part, ticket, st);
  cfg.numAttrs = 1;
  for (int p = 1; p < OC_PASSES; ++p)
    cudaLaunchKernelEx(&cfg, p == 1 ? k_oc_bisect<1> : k_oc_bisect<2>, n, rho, dr, A, vol, vf, move, ocp, part, ticket, st);
  cudaLaunchKernelEx(&cfg, k_oc_design, n, rho, (const double*)ocp, move, rho_new, part, ticket, st, host);
  return OC_PASSES + 1;
}

int oc_batch_launch(const BatchOcDesc* D, int nprob, unsigned* queue, double move, double* lam_out, int* steps_out,
                    cudaStream_t stream) {
  int dev = 0, sms = 1;  // 128 registers a thread: one block per SM
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  k_oc_batch<<<std::max(1, std::min(nprob, sms)), OCB_THREADS, 0, stream>>>(D, nprob, queue, move, lam_out, steps_out);
  return 1;
}

// ------------------------------------------------------------------ density filter
// Element arrays are in the reference's element order: axes (slowest, middle, fastest) = (x, y, z)
// in 3-D and, with a slowest axis of one element, (-, x, y) in 2-D.
struct FGrid {
  int n0, n1, n2;
};
static FGrid filter_grid(const Geo& g) {
  if (g.dim == 3) return {g.nx - 1, g.ny - 1, g.nz - 1};
  return {1, g.nx - 1, g.ny - 1};
}

// What an element does with its filtered value.
struct FoStore {
  double* out;
  EDGE_D void operator()(long long e, int, int, int, double v) const { out[e] = v; }
};
struct FoLaw {  // rho_f = H rho and E = clip(rho_f^p, void, 1) at the element's slot
  FilterOut o;
  EDGE_D void operator()(long long e, int i0, int i1, int i2, double rf) const {
    o.rho_f[e] = rf;
    const double Ev = fmin(fmax(pow(rf, o.penalty), o.vmin), 1.0);
    const long long s = o.slots.dim == 3 ? o.slots.slot3(i0, i1, i2) : o.slots.slot2(i1, i2);
    o.E64[s] = Ev;
    if (o.E32) o.E32[s] = (float)Ev;
  }
};

// Tiled filter: a block of 256 threads owns 4 x 16 x 32 elements (slowest, middle, fastest; 1 x 32 x 32
// in 2-D), stages them with a halo of the taps' reach R in shared memory (zero outside the grid; eight
// loads of a thread in flight at a time) and each thread forms four consecutive outputs along the
// middle axis per slowest position: a column of taps costs 4 + 2 R shared loads for its up to
// 4 (2 R + 1) products, and no product tests a bound.  The columns are unrolled over the whole
// (2 R + 1)^2 window, so weights are immediate constant-bank operands; a tap that the filter does not
// have is skipped (not multiplied by zero: its element may hold an infinity).
//
// Forward: sum_k w_k rho_{e+o_k} / N_e; N_e is one constant unless a tap of the element leaves the
// grid.  Transpose: sum_k w_k (v / N)_{e+o_k}, the quotients formed once while staging (the
// one-thread-per-element kernel divides w_k by N for every tap).
//
// 128 x 64 x 64, r_min 2 (27 taps), forward and transpose through the Python calls: 61.5 us with one
// thread per element, 23.3 tiled, of which the two calls' host path is 20; 400 x 200, r_min 2.5: 24.5 and
// 24.0 (host path).  Cold caches, per kernel: 12.5 us at 128 x 64 x 64, 44 at 256 x 128 x 128 (HBM floor
// 10): the fill of the halo (1.9 x the elements) and 13.5 shared loads per output.
constexpr int FT_THREADS = 256;
// The taps of a reach of R as the kernel's parameter: column (o0, o2) at [(o0 + R0) (2 R + 1) + o2 + R],
// weight of middle offset b - R at [b], bit b of present: the filter has that tap.
template <int R, int R0> struct TapParam {
  static constexpr int NC = (2 * R0 + 1) * (2 * R + 1);
  double nint;
  double w[NC][2 * R + 1];
  unsigned char present[NC];
};
template <int R, int R0> static TapParam<R, R0> tap_param(const TapCols& c) {
  TapParam<R, R0> p{};
  p.nint = c.nint;
  for (int q = 0; q < c.n; ++q) {
    const int k = (c.o0[q] + R0) * (2 * R + 1) + c.o2[q] + R;
    p.present[k] = c.present[q];
    for (int b = 0; b <= 2 * R; ++b) p.w[k][b] = c.w[q][b];
  }
  return p;
}
template <int R, int R0> struct FTile {
  static constexpr int S0 = R0 > 0 ? 4 : 1, S1 = R0 > 0 ? 16 : 32, S2 = 32;  // outputs
  static constexpr int H0 = S0 + 2 * R0, H1 = S1 + 2 * R, H2 = S2 + 2 * R;    // with halo
  static constexpr int BYTES = H0 * H1 * H2 * 8;
};

template <int R, int R0, bool TRANSPOSE, class Out>
__global__ void __launch_bounds__(FT_THREADS)
k_filter_tile(const FGrid g, const __grid_constant__ TapParam<R, R0> tc, const double* __restrict__ N,
              const double* __restrict__ in, const Out out) {
  EDGE_PDL_ENTRY();
  using T = FTile<R, R0>;
  __shared__ double sh[T::H0 * T::H1 * T::H2];
  const int b2 = blockIdx.x * T::S2, b1 = blockIdx.y * T::S1, b0 = blockIdx.z * T::S0;
  const long long p0 = (long long)g.n1 * g.n2;
  constexpr int HN = T::H0 * T::H1 * T::H2, U = 8;
  for (int q0 = threadIdx.x; q0 < HN; q0 += U * FT_THREADS) {
    double v[U], nn[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int q = q0 + k * FT_THREADS;
      const int h2 = q % T::H2, h1 = (q / T::H2) % T::H1, h0 = q / (T::H2 * T::H1);
      const int i2 = b2 + h2 - R, i1 = b1 + h1 - R, i0 = b0 + h0 - R0;
      v[k] = 0.0;
      nn[k] = tc.nint;
      if (q < HN && i2 >= 0 && i2 < g.n2 && i1 >= 0 && i1 < g.n1 && i0 >= 0 && i0 < g.n0) {
        const long long e = i0 * p0 + (long long)i1 * g.n2 + i2;
        v[k] = __ldg(in + e);
        if constexpr (TRANSPOSE) {
          if (!(i2 >= R && i2 < g.n2 - R && i1 >= R && i1 < g.n1 - R && i0 >= R0 && i0 < g.n0 - R0))
            nn[k] = __ldg(N + e);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k)
      if (q0 + k * FT_THREADS < HN) sh[q0 + k * FT_THREADS] = TRANSPOSE ? v[k] / nn[k] : v[k];
  }
  __syncthreads();
  const int l2 = threadIdx.x & 31, w = threadIdx.x >> 5;
  // 8 warps: groups of four outputs along the middle axis, then the slowest positions
  constexpr int G1 = T::S1 / 4;                          // 4 (3-D) or 8 (2-D)
  constexpr int STEP0 = 8 / G1, NL = (T::S0 + STEP0 - 1) / STEP0;  // slowest positions of a thread: l0 = f0 + STEP0 k
  const int l1 = (w % G1) * 4, f0 = w / G1;
  double acc[NL][4];
#pragma unroll
  for (int k = 0; k < NL; ++k)
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[k][a] = 0.0;
  const double* base = sh + ((f0 + R0) * T::H1 + l1) * T::H2 + l2 + R;
#pragma unroll
  for (int o0 = -R0; o0 <= R0; ++o0)
#pragma unroll
    for (int o2 = -R; o2 <= R; ++o2) {
      constexpr int W2 = 2 * R + 1;
      const int c = (o0 + R0) * W2 + o2 + R;
      const unsigned m = tc.present[c];
      if (m == 0) continue;
#pragma unroll
      for (int k = 0; k < NL; ++k) {
        double x[4 + 2 * R];
#pragma unroll
        for (int j = 0; j < 4 + 2 * R; ++j) x[j] = base[((k * STEP0 + o0) * T::H1 + j) * T::H2 + o2];
#pragma unroll
        for (int b = 0; b < W2; ++b)
          if ((m >> b) & 1)
#pragma unroll
            for (int a = 0; a < 4; ++a) acc[k][a] = fma(tc.w[c][b], x[a + b], acc[k][a]);
      }
    }
  const int i2 = b2 + l2;
  if (i2 >= g.n2) return;
#pragma unroll
  for (int k = 0; k < NL; ++k) {
    const int i0 = b0 + f0 + k * STEP0;
    if (i0 >= g.n0) break;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i1 = b1 + l1 + a;
      if (i1 >= g.n1) break;
      const long long e = i0 * p0 + (long long)i1 * g.n2 + i2;
      double v = acc[k][a];
      if constexpr (!TRANSPOSE) {
        const bool inner = i2 >= R && i2 < g.n2 - R && i1 >= R && i1 < g.n1 - R && i0 >= R0 && i0 < g.n0 - R0;
        const double nn = inner ? tc.nint : __ldg(N + e);
        v = nn > 0.0 ? v / nn : 0.0;
      }
      out(e, i0, i1, i2, v);
    }
  }
}

// One thread per element: taps that reach further than the tiles' halo.
template <int MODE, class Out>  // 0 forward, 1 transpose, 2 normaliser
__global__ void k_filter_elem(const FGrid g, const __grid_constant__ Taps taps, int dim, const double* __restrict__ N,
                              const double* __restrict__ in, const Out out) {
  EDGE_PDL_ENTRY();
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= (long long)g.n0 * g.n1 * g.n2) return;
  const int i2 = (int)(e % g.n2), i1 = (int)((e / g.n2) % g.n1), i0 = (int)(e / ((long long)g.n2 * g.n1));
  const int sh = dim == 3 ? 0 : 1;  // 2-D taps (dx, dy) are (middle, fastest)
  double sv = 0.0, sw = 0.0;
  for (int t = 0; t < taps.n; ++t) {
    const int j0 = i0 + (sh ? 0 : taps.off[t][0]), j1 = i1 + taps.off[t][1 - sh], j2 = i2 + taps.off[t][2 - sh];
    if (j0 < 0 || j0 >= g.n0 || j1 < 0 || j1 >= g.n1 || j2 < 0 || j2 >= g.n2) continue;
    const long long q = ((long long)j0 * g.n1 + j1) * g.n2 + j2;
    const double w = taps.w[t];
    if constexpr (MODE == 0) sv += w * __ldg(in + q);
    if constexpr (MODE == 1) sv += (w / __ldg(N + q)) * __ldg(in + q);
    sw += w;
  }
  if constexpr (MODE == 0) out(e, i0, i1, i2, sw > 0.0 ? sv / sw : 0.0);
  if constexpr (MODE == 1) out(e, i0, i1, i2, sv);
  if constexpr (MODE == 2) out(e, i0, i1, i2, sw);
}

bool make_tap_cols(int dim, const Taps& t, TapCols& c) {
  c = TapCols{};
  for (int k = 0; k < t.n; ++k) {
    const int o0 = dim == 3 ? t.off[k][0] : 0, o1 = dim == 3 ? t.off[k][1] : t.off[k][0],
              o2 = dim == 3 ? t.off[k][2] : t.off[k][1];
    if (std::abs(o0) > FT_RMAX || std::abs(o1) > FT_RMAX || std::abs(o2) > FT_RMAX) return false;
    if (dim == 2 && t.off[k][2] != 0) return false;
    c.R = std::max({c.R, std::abs(o1), std::abs(o2), std::abs(o0), 1});
    c.R0 = dim == 3 ? 1 : 0;
    c.nint += t.w[k];
  }
  for (int k = 0; k < t.n; ++k) {
    const int o0 = dim == 3 ? t.off[k][0] : 0, o1 = dim == 3 ? t.off[k][1] : t.off[k][0],
              o2 = dim == 3 ? t.off[k][2] : t.off[k][1];
    int q = 0;
    while (q < c.n && !(c.o0[q] == o0 && c.o2[q] == o2)) ++q;
    if (q == c.n) {
      if (c.n == FT_COLS) return false;
      c.o0[q] = (signed char)o0;
      c.o2[q] = (signed char)o2;
      ++c.n;
    }
    const int b = o1 + c.R;
    if ((c.present[q] >> b) & 1) return false;  // a repeated offset
    c.present[q] |= (unsigned char)(1u << b);
    c.w[q][b] = t.w[k];
  }
  return c.n > 0;
}

template <int R, int R0, bool TR, class Out>
static int filter_tile_launch(const FGrid& g, const TapCols& c, const double* N, const double* in, const Out& out,
                              cudaStream_t stream) {
  using T = FTile<R, R0>;
  static_assert(T::BYTES <= 48 * 1024, "static shared memory");
  auto up = [](int a, int b) { return (unsigned)((a + b - 1) / b); };
  k_filter_tile<R, R0, TR, Out><<<dim3(up(g.n2, T::S2), up(g.n1, T::S1), up(g.n0, T::S0)), FT_THREADS, 0, stream>>>(
      g, tap_param<R, R0>(c), N, in, out);
  return 1;
}
// Reaches 1 and 2 (r_min up to 3 on equal edges) and 3 in 2-D are tiled; the tile counts of the middle
// and slowest axes are grid dimensions y and z (limit 65,535).
template <bool TR, class Out>
static int filter_run(const Geo& geo, const Taps& t, const TapCols* c, const double* N, const double* in, const Out& out,
                      cudaStream_t stream) {
  const FGrid g = filter_grid(geo);
  if (c && g.n1 <= 65535 * 16 && g.n0 <= 65535 * 4) {
    if (c->R0 == 0) {
      switch (c->R) {
        case 1: return filter_tile_launch<1, 0, TR, Out>(g, *c, N, in, out, stream);
        case 2: return filter_tile_launch<2, 0, TR, Out>(g, *c, N, in, out, stream);
        default: return filter_tile_launch<3, 0, TR, Out>(g, *c, N, in, out, stream);
      }
    }
    if (c->R == 1) return filter_tile_launch<1, 1, TR, Out>(g, *c, N, in, out, stream);
    if (c->R == 2) return filter_tile_launch<2, 2, TR, Out>(g, *c, N, in, out, stream);
  }
  const long long n = (long long)g.n0 * g.n1 * g.n2;
  k_filter_elem<TR ? 1 : 0, Out><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(g, t, geo.dim, N, in, out);
  return 1;
}

int filter_forward(const Geo& g, const Taps& t, const TapCols* c, const double* N, const double* in,
                   const FilterOut& out, cudaStream_t stream) {
  if (out.E64) return filter_run<false>(g, t, c, N, in, FoLaw{out}, stream);
  return filter_run<false>(g, t, c, N, in, FoStore{out.rho_f}, stream);
}
int filter_transpose(const Geo& g, const Taps& t, const TapCols* c, const double* N, const double* in, double* out,
                     cudaStream_t stream) {
  return filter_run<true>(g, t, c, N, in, FoStore{out}, stream);
}
int filter_norm(const Geo& g, const Taps& t, double* N, cudaStream_t stream) {
  const FGrid f = filter_grid(g);
  const long long n = (long long)f.n0 * f.n1 * f.n2;
  k_filter_elem<2, FoStore><<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(f, t, g.dim, nullptr, nullptr, FoStore{N});
  return 1;
}

// ------------------------------------------------------------------ operator on user vectors, 2-D
// K(E) u straight from and to the user's interleaved vectors: one launch instead of the conversion
// to slots, the tiled product and the conversion back.  One thread per node gathers its nine
// neighbours (16-byte pairs where the vector is 16-byte aligned; a neighbour outside the grid reads
// the node itself and counts as zero, so that all loads of a thread are in flight together) and the
// four surrounding elements, 64 FMA with the element matrix in the constant bank.  What bounds it
// is the launch and two round trips to L2: at 131,841 nodes the FMA take 0.5 us.
template <bool PAIR> EDGE_D double2 user_pair(const double* __restrict__ u, long long node) {
  if constexpr (PAIR) return __ldg(reinterpret_cast<const double2*>(u) + node);
  else return make_double2(__ldg(u + 2 * node), __ldg(u + 2 * node + 1));
}
template <bool PAIR>
__global__ void __launch_bounds__(128)
k_product2_user(const Geo g, const __grid_constant__ K2Dense K, const double* __restrict__ E,
                const uint8_t* __restrict__ mask, const double* __restrict__ u, double* __restrict__ out) {
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), j = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (i >= g.nx || j >= g.ny) return;
  const long long node = (long long)j * g.nx + i, s = g.slot2(i, j);
  double U[3][3][2], Ee[2][2];
  double2 raw = make_double2(0.0, 0.0);
  unsigned mc = 0;
#pragma unroll
  for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
    for (int dx = -1; dx <= 1; ++dx) {
      const bool in = i + dx >= 0 && i + dx < g.nx && j + dy >= 0 && j + dy < g.ny;
      const double2 v = user_pair<PAIR>(u, in ? node + (long long)dy * g.nx + dx : node);
      const unsigned m = in ? __ldg(mask + s + (long long)dy * g.pz + dx) : 3u;
      if (dx == 0 && dy == 0) {
        raw = v;
        mc = m;
      }
      U[dy + 1][dx + 1][0] = (m & 1) ? 0.0 : v.x;
      U[dy + 1][dx + 1][1] = (m & 2) ? 0.0 : v.y;
    }
#pragma unroll
  for (int ay = 0; ay < 2; ++ay)
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {  // the element of which the node is corner (ax, ay)
      const int li = i - ax, lj = j - ay;
      const bool ev = li >= 0 && lj >= 0 && li < g.nx - 1 && lj < g.ny - 1;
      const double x = __ldg(E + (ev ? g.slot2(li, lj) : s));
      Ee[ay][ax] = ev ? x : 0.0;
    }
  double A0 = 0.0, A1 = 0.0;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int ax = a & 1, ay = a >> 1;
    double r0 = 0.0, r1 = 0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const double ub = U[(b >> 1) - ay + 1][(b & 1) - ax + 1][d];
        r0 = fma(K.k[(a * 2 + 0) * 8 + b * 2 + d], ub, r0);
        r1 = fma(K.k[(a * 2 + 1) * 8 + b * 2 + d], ub, r1);
      }
    A0 = fma(Ee[ay][ax], r0, A0);
    A1 = fma(Ee[ay][ax], r1, A1);
  }
  if (mc & 1) A0 = raw.x;
  if (mc & 2) A1 = raw.y;
  if constexpr (PAIR) {
    reinterpret_cast<double2*>(out)[node] = make_double2(A0, A1);
  } else {
    out[2 * node] = A0;
    out[2 * node + 1] = A1;
  }
}

// Element energies: elements run along y in the reference's order, nodes along x, so a block stages
// the 33 x 33 nodes of 32 x 32 elements (rows along x, coalesced) and its lanes then walk elements
// along y (coalesced stores; the row pitch of 33 pairs keeps eight lanes on different banks).
EDGE_D double energy2(const KHat2<double>& K, const double u[4][2]) { return elem2_energy(K, u); }
EDGE_D double energy2(const K2Dense& K, const double u[4][2]) {
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += K.k[r * 8 + q] * u[q >> 1][q & 1];
    acc += u[r >> 1][r & 1] * t;
  }
  return acc;
}
template <bool PAIR, class K2>
__global__ void __launch_bounds__(256)
k_energy2_user(const Geo g, const __grid_constant__ K2 K, const double* __restrict__ u, double* __restrict__ dk) {
  __shared__ double2 sh[33 * 33];
  const int nelx = g.nx - 1, nely = g.ny - 1;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  constexpr int U = 5;  // 33 * 33 nodes over 256 threads
  double2 v[U];
#pragma unroll
  for (int k = 0; k < U; ++k) {
    const int q = threadIdx.x + k * 256, i = x0 + q % 33, j = y0 + q / 33;
    const bool in = q < 33 * 33 && i < g.nx && j < g.ny;
    v[k] = in ? user_pair<PAIR>(u, (long long)j * g.nx + i) : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (threadIdx.x + k * 256 < 33 * 33) sh[threadIdx.x + k * 256] = v[k];
  __syncthreads();
  const int ly = threadIdx.x & 31, j = y0 + ly;
  if (j >= nely) return;
  for (int lx = threadIdx.x >> 5; lx < 32; lx += 8) {
    const int i = x0 + lx;
    if (i >= nelx) break;
    double ue[4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const double2 p = sh[(ly + (b >> 1)) * 33 + lx + (b & 1)];
      ue[b][0] = p.x;
      ue[b][1] = p.y;
    }
    dk[(long long)i * nely + j] = -energy2(K, ue);
  }
}

static bool pair_aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }

int product2_user(const Geo& g, const K2Dense& K, const double* E, const uint8_t* mask, const double* u, double* out,
                  cudaStream_t stream) {
  const dim3 grid((g.nx + 31) / 32, (g.ny + 3) / 4);
  if (pair_aligned(u) && pair_aligned(out))
    k_product2_user<true><<<grid, 128, 0, stream>>>(g, K, E, mask, u, out);
  else
    k_product2_user<false><<<grid, 128, 0, stream>>>(g, K, E, mask, u, out);
  return 1;
}
template <class K2>
static int energy2_launch(const Geo& g, const K2& K, const double* u, double* dk, cudaStream_t stream) {
  const dim3 grid((g.nx - 1 + 31) / 32, (g.ny - 1 + 31) / 32);
  if (pair_aligned(u))
    k_energy2_user<true, K2><<<grid, 256, 0, stream>>>(g, K, u, dk);
  else
    k_energy2_user<false, K2><<<grid, 256, 0, stream>>>(g, K, u, dk);
  return 1;
}
int energy2_user(const Geo& g, const K2Dense& K, const KHat2<double>* box, const double* u, double* dk,
                 cudaStream_t stream) {
  return box ? energy2_launch(g, *box, u, dk, stream) : energy2_launch(g, K, u, dk, stream);
}

// ------------------------------------------------------------------ operator on user vectors, 3-D
// K(E) u (or the element energies u_e^T K0 u_e) straight from the user's interleaved vector, FP64.
// The walk is the one of the TMA kernel (fine_tma.cuh): 4 warps of 16 z-lanes x 2 x-columns march
// along y with one element per thread and layer, in the Walsh transform domain.  A user row (3 nz
// doubles) has no 16-byte pitch, so planes arrive by 8-byte cp.async copies into a four-stage ring
// (zero-filled outside the grid), each thread copying the same four positions of every plane; E and the
// constraint flags of a layer are fetched one layer ahead.  The in-plane sums of neighbouring warps
// are exchanged through shared memory and picked up one layer later, so that a layer has one
// barrier; outputs are gathered per warp and stored contiguously.
//
// Layers are unrolled by four: stages are constants and the lower and upper plane swap without copies
// (103M warp instructions at 12.8M DOF rolled, 61M unrolled).
//
// What bounds it: FP64 latency at 12 warps per SM.  An element takes 150 FP64 operations (200 without
// the cube's block form): 45 us of the FP64 pipe at 12.8M DOF with the tiles' overlap, 37 us for the
// bytes; it runs in 134.  Blocks of 4 warps at 168 registers, three per SM, measured best: 8 warps at
// 128 registers 144 us (spills), four blocks 152 (spills), two 167.  (Without the block form the product
// spills 48 bytes at 168 registers.)  The three launches it replaces
// (user to slots, TMA product, slots to user) took 205 us.
constexpr int U3_BX = 4, U3_NS = 4;
constexpr int U3_NC = 2 * U3_BX, U3_NR = U3_NC + 1, U3_ROW = 51;  // element columns, node rows, doubles per row
constexpr int U3_PLANE = U3_NR * U3_ROW, U3_PER = (U3_PLANE + 127) / 128;

EDGE_D void cp_async8(void* dst, const void* src, bool valid) {
  const int n = valid ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(n)
               : "memory");
}
EDGE_D void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> EDGE_D void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// v = E Khat u for h = 1..7 (h = 0 is neither read nor written).
EDGE_D void khat3(const KHat3<double>& K, double E, const double u[8][3], double v[8][3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int h = 1; h < 8; ++h) {
      double a = K.dg[c][h] * u[h][c];
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (d != c && (((h >> c) & 1) != ((h >> d) & 1))) a = fma(K.of[c][d][h], u[h ^ (1 << c) ^ (1 << d)][d], a);
      v[h][c] = a * E;
    }
}
EDGE_D void khat3(const KCube64& k, double E, const double u[8][3], double v[8][3]) {
  const double nd = k.nd * E, no = k.no * E, sh = k.sh * E, bd = k.bd * E, bo = k.bo * E, td = k.td * E, to = k.to * E,
               h7 = k.h7 * E;
  const double ns = no * (u[1][0] + u[2][1] + u[4][2]);  // normal strains
  v[1][0] = fma(nd, u[1][0], ns);
  v[2][1] = fma(nd, u[2][1], ns);
  v[4][2] = fma(nd, u[4][2], ns);
  const double ts = to * (u[3][2] + u[5][1] + u[6][0]);  // twists
  v[3][2] = fma(td, u[3][2], ts);
  v[5][1] = fma(td, u[5][1], ts);
  v[6][0] = fma(td, u[6][0], ts);
  v[1][1] = v[2][0] = sh * (u[1][1] + u[2][0]);  // shears
  v[1][2] = v[4][0] = sh * (u[1][2] + u[4][0]);
  v[2][2] = v[4][1] = sh * (u[2][2] + u[4][1]);
  v[3][0] = fma(bd, u[3][0], bo * u[6][2]);  // bending pairs
  v[6][2] = fma(bd, u[6][2], bo * u[3][0]);
  v[3][1] = fma(bd, u[3][1], bo * u[5][2]);
  v[5][2] = fma(bd, u[5][2], bo * u[3][1]);
  v[5][0] = fma(bd, u[5][0], bo * u[6][1]);
  v[6][1] = fma(bd, u[6][1], bo * u[5][0]);
#pragma unroll
  for (int c = 0; c < 3; ++c) v[7][c] = h7 * u[7][c];
}
EDGE_D void wht_plane(double t[2][2][3]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const double p = t[b][0][c], q = t[b][1][c];
      t[b][0][c] = p + q;
      t[b][1][c] = p - q;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double p = t[0][h][c], q = t[1][h][c];
      t[0][h][c] = p + q;
      t[1][h][c] = p - q;
    }
  }
}

template <bool PRODUCT, class K3>
__global__ void __launch_bounds__(32 * U3_BX, 3)
k_user3(const Geo g, const __grid_constant__ K3 K, const double* __restrict__ E, const uint8_t* __restrict__ mask,
        const uint8_t* __restrict__ eflag16, const int mpz, const int ly, const double* __restrict__ u,
        double* __restrict__ out) {
  __shared__ double sP[U3_NS][U3_PLANE];
  __shared__ double sX[PRODUCT ? 2 : 1][PRODUCT ? U3_BX : 1][16][3];
  __shared__ double sO[PRODUCT ? U3_BX : 1][2][48];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int zl = lane & 15, xh = lane >> 4, cx = 2 * w + xh;
  // first node column / z of the tile: one before the outputs for the product
  const int tz = PRODUCT ? (int)blockIdx.x * 15 - 1 : (int)blockIdx.x * 16;
  const int tx = PRODUCT ? (int)blockIdx.y * (U3_NC - 1) - 1 : (int)blockIdx.y * U3_NC;
  const int rows = PRODUCT ? g.ny : g.ny - 1;  // output planes / element rows
  const int y0 = blockIdx.z * ly, y1 = min(y0 + ly, rows);
  const int p0 = PRODUCT ? y0 - 1 : y0, np = y1 - p0 + 1;
  const int ez = tz + zl, ex = tx + cx;

  // the positions of a plane that this thread copies, as one pointer that moves a plane per copy
  int off[U3_PER];
  bool ok[U3_PER];
#pragma unroll
  for (int t = 0; t < U3_PER; ++t) {
    const int q = threadIdx.x + t * (32 * U3_BX), r = q / U3_ROW, c = q % U3_ROW;
    const int x = tx + r, z = tz + c / 3;
    ok[t] = q < U3_PLANE && x >= 0 && x < g.nx && z >= 0 && z < g.nz;
    off[t] = ok[t] ? (x * g.nz + z) * 3 + c % 3 : 0;
  }
  const long long pl = 3LL * g.nx * g.nz;
  const double* src = u + p0 * pl;  // plane p0 + (next k); dereferenced only inside the grid
  int pk = p0;
  auto issue = [&](int stage) {
    const bool in = pk >= 0 && pk < g.ny && pk <= y1;
    const double* from = in ? src : u;
#pragma unroll
    for (int t = 0; t < U3_PER; ++t)
      if (t + 1 < U3_PER || threadIdx.x + t * (32 * U3_BX) < U3_PLANE)
        cp_async8(sP[stage] + threadIdx.x + t * (32 * U3_BX), from + off[t], in && ok[t]);
    cp_commit();
    src += pl;
    ++pk;
  };
  const bool col = ex >= 0 && ex < g.nx && ez >= 0 && ez < g.nz;
  // E and the constraint flag of this thread's column, one plane of slots per step
  const double* Ep = PRODUCT && col ? E + g.slot3(ex, 0, ez) : nullptr;
  const uint8_t* Fp = PRODUCT && col ? eflag16 + (long long)ex * mpz + ez : nullptr;
  const long long fpl = (long long)g.nx * mpz;
  auto elem_E = [&](int ey) -> double { return col && (unsigned)ey < (unsigned)g.ny ? __ldg(Ep + ey * g.plane) : 0.0; };
  auto elem_flag = [&](int ey) -> unsigned {
    return col && (unsigned)ey < (unsigned)g.ny ? __ldg(Fp + ey * fpl) : 0u;
  };
  // constrained DOFs of the four corners on plane p read as zero (flagged columns: ex, ez >= 0)
  auto mask_plane = [&](int p, double t[2][2][3]) {
#pragma unroll
    for (int dx = 0; dx < 2; ++dx)
#pragma unroll
      for (int dz = 0; dz < 2; ++dz)
        if (ex + dx < g.nx && ez + dz < g.nz && p >= 0 && p < g.ny) {
          const unsigned m = __ldg(mask + g.slot3(ex + dx, p, ez + dz));
#pragma unroll
          for (int c = 0; c < 3; ++c)
            if ((m >> c) & 1) t[dx][dz][c] = 0.0;
        }
  };
  const double* corner = sP[0] + cx * U3_ROW + 3 * zl;
  auto load_plane = [&](int stage, double t[2][2][3]) {
#pragma unroll
    for (int dx = 0; dx < 2; ++dx)
#pragma unroll
      for (int dz = 0; dz < 2; ++dz)
#pragma unroll
        for (int c = 0; c < 3; ++c) t[dx][dz][c] = corner[stage * U3_PLANE + dx * U3_ROW + 3 * dz + c];
  };

#pragma unroll
  for (int k = 0; k < U3_NS - 1; ++k) issue(k);
  // E and flags of the coming layers, fetched two layers before they are used
  double Ee = PRODUCT ? elem_E(p0) : 1.0, E1 = PRODUCT ? elem_E(p0 + 1) : 1.0;
  unsigned fl = PRODUCT ? elem_flag(p0) : 0u, fn = PRODUCT ? elem_flag(p0 + 1) : 0u, f2 = PRODUCT ? elem_flag(p0 + 2) : 0u;
  cp_wait<U3_NS - 2>();
  __syncthreads();
  double pa[2][2][3], pb[2][2][3], car[2][2][3], pend[3];
  load_plane(0, pa);
  if (PRODUCT && fl) mask_plane(p0, pa);
  wht_plane(pa);
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int c = 0; c < 3; ++c) car[a][b][c] = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) pend[c] = 0.0;
  unsigned pfl = 0;
  // this lane's three places of the warp half's output row (16 nodes from z = tz), moving a plane per
  // store
  bool st[3];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const int d = zl + 16 * t;
    st[t] = PRODUCT && cx >= 1 && ex < g.nx && d >= 3 && tz + d / 3 < g.nz;
  }
  double* op = out + (((long long)y0 * g.nx + ex) * g.nz + tz) * 3 + zl;  // dereferenced only where st

  // completes and stores plane p, the output of the layer before; X: its exchange buffer
  auto flush = [&](int p, int X) {
    double a[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = pend[c];
    if (xh == 0 && w > 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a[c] += sX[X][w - 1][zl][c];
    }
    if (pfl && zl >= 1 && cx >= 1) {  // identity rows
      const unsigned m = __ldg(mask + g.slot3(ex, p, ez));
      const long long node = ((long long)p * g.nx + ex) * g.nz + ez;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        if ((m >> c) & 1) a[c] = __ldg(u + 3 * node + c);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) sO[w][xh][3 * zl + c] = a[c];
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 3; ++t)
      if (st[t]) op[16 * t] = sO[w][xh][zl + 16 * t];
    op += pl;
  };

  // one layer: element row ey between the planes lo (transformed) and the one in stage S
  auto layer = [&](int ey, auto stage, double lo[2][2][3], double hi[2][2][3]) {
    constexpr int S = decltype(stage)::value;  // the new plane's stage = (layer + 1) mod 4
    cp_wait<U3_NS - 3>();
    __syncthreads();
    issue((S + U3_NS - 2) % U3_NS);
    double E2 = 1.0;
    unsigned f3 = 0u;
    if constexpr (PRODUCT) {
      E2 = elem_E(ey + 2);
      f3 = elem_flag(ey + 3);
      if (ey > y0) flush(ey - 1, S & 1);
    }
    load_plane(S, hi);
    // the new plane is also the lower face of the next element row: masked by both rows' flags
    if (PRODUCT && (fl | fn)) mask_plane(ey + 1, hi);
    wht_plane(hi);
    double uh[8][3], vh[8][3];
#pragma unroll
    for (int hx = 0; hx < 2; ++hx)
#pragma unroll
      for (int hz = 0; hz < 2; ++hz)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (hx | hz) uh[hx | (hz << 2)][c] = lo[hx][hz][c] + hi[hx][hz][c];
          uh[hx | 2 | (hz << 2)][c] = lo[hx][hz][c] - hi[hx][hz][c];
        }
    khat3(K, Ee, uh, vh);
    if constexpr (PRODUCT) {
      double cur[2][2][3];
#pragma unroll
      for (int hx = 0; hx < 2; ++hx)
#pragma unroll
        for (int hz = 0; hz < 2; ++hz)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const double b = vh[hx | 2 | (hz << 2)][c];
            if (hx | hz) {
              const double a = vh[hx | (hz << 2)][c];
              cur[hx][hz][c] = car[hx][hz][c] + (a + b);
              car[hx][hz][c] = a - b;
            } else {  // transform coefficient 0 vanishes
              cur[0][0][c] = car[0][0][c] + b;
              car[0][0][c] = -b;
            }
          }
      wht_plane(cur);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const double g0 = cur[0][0][c] + __shfl_up_sync(0xffffffffu, cur[0][1][c], 1, 16);
        const double g1 = cur[1][0][c] + __shfl_up_sync(0xffffffffu, cur[1][1][c], 1, 16);
        const double fromL = __shfl_up_sync(0xffffffffu, g1, 16);
        pend[c] = xh ? g0 + fromL : g0;
        if (xh) sX[(S + 1) & 1][w][zl][c] = g1;
      }
      pfl = fl;
    } else {
      double e = 0.0;
#pragma unroll
      for (int h = 1; h < 8; ++h)
#pragma unroll
        for (int c = 0; c < 3; ++c) e = fma(uh[h][c], vh[h][c], e);
      if (ex < g.nx - 1 && ez < g.nz - 1) out[((long long)ex * (g.ny - 1) + ey) * (g.nz - 1) + ez] = -e;
    }
    Ee = E1;
    E1 = E2;
    fl = fn;
    fn = f2;
    f2 = f3;
  };
  // layers in groups of four: the stage is then a constant and the two planes swap without copies
  int ey = p0;
  const int last = p0 + np - 1;  // one past the last element row
  int done = 0;
  for (; ey + 4 <= last; ey += 4) {
    layer(ey, std::integral_constant<int, 1>{}, pa, pb);
    layer(ey + 1, std::integral_constant<int, 2>{}, pb, pa);
    layer(ey + 2, std::integral_constant<int, 3>{}, pa, pb);
    layer(ey + 3, std::integral_constant<int, 0>{}, pb, pa);
  }
  if (ey < last) {
    layer(ey, std::integral_constant<int, 1>{}, pa, pb);
    done = 1;
  }
  if (ey + 1 < last) {
    layer(ey + 1, std::integral_constant<int, 2>{}, pb, pa);
    done = 2;
  }
  if (ey + 2 < last) {
    layer(ey + 2, std::integral_constant<int, 3>{}, pa, pb);
    done = 3;
  }
  if constexpr (PRODUCT) {
    __syncthreads();
    flush(last - 1, (done + 1) & 1);  // the last layer wrote buffer (its stage + 1) & 1
  }
  cp_wait<0>();
}

// Tiles of k_user3 along z and x and the rows it marches over: product tiles overlap by one element.
struct User3Tiles {
  long long tz, tx;
  int rows;
};
static User3Tiles user3_tiles(const Geo& g, bool product) {
  auto up = [](int n, int step) { return (long long)(n + step - 1) / step; };
  if (product) return {up(g.nz, 15), up(g.nx, U3_NC - 1), g.ny};
  return {up(g.nz - 1, 16), up(g.nx - 1, U3_NC), g.ny - 1};
}

// Rows per block: the number of y-chunks that needs the fewest layers in all, counting the waves of
// resident blocks (three per SM) and one and a half layers of start-up per block.  Up to 4,096
// candidates: a plan of the grid, made once with the problem (made in every call, the energies of
// 8 x 4,000 x 8 elements took 18.8 us instead of 8.8).
int user3_rows(const Geo& g, bool product) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const User3Tiles t = user3_tiles(g, product);
  const long long tiles = t.tz * t.tx, wave = 3LL * sms;
  long long best = -1;
  int best_ly = t.rows;
  for (int c = 1; c <= t.rows && c <= 4096; ++c) {
    const int ly = (t.rows + c - 1) / c;
    const long long blocks = tiles * ((t.rows + ly - 1) / ly);
    const long long cost = ((blocks + wave - 1) / wave) * (2LL * ly + 3);
    if (best < 0 || cost < best) {
      best = cost;
      best_ly = ly;
    }
    if (tiles * c > wave * 64) break;
  }
  return best_ly;
}

bool user_grid_ok(const Geo& g, bool product) {
  constexpr int MAX_YZ = 65535;  // grid dimensions y and z
  if (g.dim == 2) return (g.ny + 3) / 4 <= MAX_YZ;
  return 3LL * g.nx * g.nz < (1LL << 31) && user3_tiles(g, product).tx <= MAX_YZ && g.ny <= MAX_YZ;
}

template <bool PRODUCT, class K3>
static int user3_launch(const Geo& g, const K3& K, const double* E, const uint8_t* mask, const uint8_t* eflag16, int mpz,
                        int ly, const double* u, double* out, cudaStream_t stream) {
  const User3Tiles t = user3_tiles(g, PRODUCT);
  const dim3 grid((unsigned)t.tz, (unsigned)t.tx, (unsigned)((t.rows + ly - 1) / ly));
  k_user3<PRODUCT, K3><<<grid, 32 * U3_BX, 0, stream>>>(g, K, E, mask, eflag16, mpz, ly, u, out);
  return 1;
}
int product3_user(const Geo& g, const KHat3<double>& K, const KCube64* cube, const double* E, const uint8_t* mask,
                  const uint8_t* eflag16, int mpz, int ly, const double* u, double* out, cudaStream_t stream) {
  if (cube) return user3_launch<true>(g, *cube, E, mask, eflag16, mpz, ly, u, out, stream);
  return user3_launch<true>(g, K, E, mask, eflag16, mpz, ly, u, out, stream);
}
int energy3_user(const Geo& g, const KHat3<double>& K, const KCube64* cube, int ly, const double* u, double* dk,
                 cudaStream_t stream) {
  if (cube) return user3_launch<false>(g, *cube, nullptr, nullptr, nullptr, 0, ly, u, dk, stream);
  return user3_launch<false>(g, K, nullptr, nullptr, nullptr, 0, ly, u, dk, stream);
}

// ------------------------------------------------------------------ coarsest level
// Inverse of the coarsest Galerkin matrix by the symmetric sweep (Gauss-Jordan) on 64 x 64 blocks: for
// every block column K, with P = A_KK^-1,
//   A_KK <- -P,   A_iK <- A_iK P,   A_ij <- A_ij - A_iK P A_Kj   (i, j != K),
// after all of which A holds -A^-1; a positive definite matrix needs no pivoting (its pivots are the
// squares of the Cholesky diagonal, checked as they come).  Only the blocks on and below the diagonal
// are kept.  Per K two launches: the panel A_iK P, and the rank-64 update of all other blocks, whose
// block (K + 1, K + 1) goes on to invert itself so that the next panel can start.  Every product is a
// 64 x 64 x 64 FP64 tile product (4 x 4 outputs per thread, operands k-major in shared memory).
//
// What bounds it: the nt = nd / 64 steps in sequence for small matrices (a block's own inverse is a
// chain of 64 sweeps, 24 us), FP64 rate (nd^3 operations) and the tiles' way through L2 for large ones:
// 0.13 ms at nd = 135 and 192, 0.46 at 675, 2.1 at 2,352, 7.3 at 4,131.  The blocked Cholesky
// factorisation with one block per column of the inverse that it replaces was a chain of 2 nd
// barrier-separated vector updates on a factor reread by every column: 13 ms at 2,352, 110 at 4,131.
constexpr int INV_T = 256;

// acc -= L R^T for k-major operands L[k][r], R[k][c], k < KD, with rows of LD doubles in shared memory
template <int KD, int LD, bool MINUS> EDGE_D void tile_mac(const double* L, const double* R, double acc[4][4]) {
  L += (threadIdx.x >> 4) * 4;
  R += (threadIdx.x & 15) * 4;
#pragma unroll 4
  for (int k = 0; k < KD; ++k, L += LD, R += LD) {
    double a[4], b[4];
    *reinterpret_cast<double2*>(a) = *reinterpret_cast<const double2*>(L);
    *reinterpret_cast<double2*>(a + 2) = *reinterpret_cast<const double2*>(L + 2);
    *reinterpret_cast<double2*>(b) = *reinterpret_cast<const double2*>(R);
    *reinterpret_cast<double2*>(b + 2) = *reinterpret_cast<const double2*>(R + 2);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma(MINUS ? -a[i] : a[i], b[j], acc[i][j]);
  }
}

// P = a^-1 of the block whose 4 x 4 pieces the threads hold: scalar sweeps a_rc <- a_rc - v_r v_c / d
// with v column k and d = v_k.  The pivot's row and column take the same update from zero with
// -1 / d in place of v_r / d and -1 in place of v_c.  One barrier per sweep: the owners of the next
// pivot's column publish it as soon as they have updated it.  sv: 2 x 64 doubles.
EDGE_D void block_invert(double a[4][4], double* sv, double* __restrict__ P, int* status) {
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  if (tx == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) sv[ty * 4 + i] = a[i][0];
  }
  __syncthreads();
  bool bad = false;
  for (int kb = 0; kb < 16; ++kb) {
    const bool mr = ty == kb, mc = tx == kb;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int k = kb * 4 + kk;
      const double* v = sv + (k & 1) * INV_B;
      double d = v[k];
      double vr[4], vc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        vr[i] = v[ty * 4 + i];
        vc[i] = v[tx * 4 + i];
      }
      if (!(d > 0.0)) {
        bad = true;
        d = 1.0;
      }
      const double inv = 1.0 / d;
      if (mr) vr[kk] = -1.0;
      if (mc) vc[kk] = -1.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) vr[i] *= inv;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (mr) a[kk][i] = 0.0;
        if (mc) a[i][kk] = 0.0;
      }
      // the next pivot's column first
      const int kn = k + 1;
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i][(kk + 1) & 3] = fma(-vr[i], vc[(kk + 1) & 3], a[i][(kk + 1) & 3]);
      if (kn < INV_B && tx == kn >> 2) {
#pragma unroll
        for (int i = 0; i < 4; ++i) sv[(kn & 1) * INV_B + ty * 4 + i] = a[i][(kk + 1) & 3];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j != ((kk + 1) & 3))
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i][j] = fma(-vr[i], vc[j], a[i][j]);
      __syncthreads();
    }
  }
  if (bad && threadIdx.x == 0) *status = 1;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) P[(ty * 4 + i) * INV_B + tx * 4 + j] = -a[i][j];
}

// Unit diagonal on the padding, and the inverse of block (0, 0).
__global__ void __launch_bounds__(INV_T) k_inv_start(double* __restrict__ A, int nd, int np, double* __restrict__ P, int* status) {
  EDGE_PDL_ENTRY();
  __shared__ double sv[2 * INV_B];
  const int r0 = (threadIdx.x >> 4) * 4, c0 = (threadIdx.x & 15) * 4;
  for (int i = nd + threadIdx.x; i < np; i += INV_T) A[(long long)i * np + i] = 1.0;
  __syncthreads();
  double a[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) a[i][j] = A[(long long)(r0 + i) * np + c0 + j];
  block_invert(a, sv, P, status);
}

// Block i of the panel: R_i = A_iK kept k-major in Rt, W_i = R_i P k-major in Wt and in A.  Shared rows
// of 66 doubles: the transposed fill meets two-way bank conflicts only.
constexpr int INV_LD = INV_B + 2;
__global__ void __launch_bounds__(INV_T)
k_inv_panel(double* __restrict__ A, int np, int K, const double* __restrict__ P, double* __restrict__ Rt, double* __restrict__ Wt) {
  EDGE_PDL_ENTRY();
  extern __shared__ __align__(16) double inv_smem[];
  double *sR = inv_smem, *sP = sR + INV_B * INV_LD;
  const int I = blockIdx.x, r0 = (threadIdx.x >> 4) * 4, c0 = (threadIdx.x & 15) * 4;
  const long long iB = (long long)I * INV_B, kB = (long long)K * INV_B;
  if (I == K) {
    for (int q = threadIdx.x; q < INV_B * INV_B; q += INV_T)
      A[(kB + q / INV_B) * np + kB + q % INV_B] = -P[q];
    return;
  }
#pragma unroll
  for (int t = 0; t < INV_B * INV_B / INV_T; ++t) {
    const int q = threadIdx.x + t * INV_T, x = q / INV_B, y = q % INV_B;
    sP[x * INV_LD + y] = P[q];
    if (I > K) sR[y * INV_LD + x] = A[(iB + x) * np + kB + y];
    else sR[x * INV_LD + y] = A[(kB + x) * np + iB + y];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < INV_B * INV_B; q += INV_T)
    Rt[(q / INV_B) * (long long)np + iB + q % INV_B] = sR[q / INV_B * INV_LD + q % INV_B];
  double acc[4][4] = {};
  tile_mac<INV_B, INV_LD, false>(sR, sP, acc);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      sR[(c0 + j) * INV_LD + r0 + i] = acc[i][j];
      if (I > K) A[(iB + r0 + i) * np + kB + c0 + j] = acc[i][j];
    }
  __syncthreads();
  for (int q = threadIdx.x; q < INV_B * INV_B; q += INV_T) {
    const int k = q / INV_B, r = q % INV_B;
    const double v = sR[k * INV_LD + r];
    Wt[k * (long long)np + iB + r] = v;
    if (I < K) A[(kB + k) * np + iB + r] = v;
  }
}

EDGE_D void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// A_ij -= W_i R_j^T for the blocks i >= j other than row and column K.  All of a tile's operands are
// requested at once (the second half of the depth arrives while the first is multiplied).  The block
// that inverts itself at the end is the first of the grid, so that this overlaps the other tiles.
__global__ void __launch_bounds__(INV_T, 3)
k_inv_update(double* __restrict__ A, int np, int K, const double* __restrict__ Rt, const double* __restrict__ Wt,
             double* __restrict__ Pnext, int* status) {
  EDGE_PDL_ENTRY();
  extern __shared__ __align__(16) double inv_smem[];
  double *sW = inv_smem, *sR = sW + INV_B * INV_B;
  int q = blockIdx.x;
  const int qd = (K + 1) * (K + 2) / 2 + K + 1;  // block (K + 1, K + 1)
  if (qd < (int)gridDim.x) q = q == 0 ? qd : q == qd ? 0 : q;
  int I = (int)((sqrtf(8.f * q + 1.f) - 1.f) * 0.5f);
  while ((I + 1) * (I + 2) / 2 <= q) ++I;
  while (I * (I + 1) / 2 > q) --I;
  const int J = q - I * (I + 1) / 2;
  if (I == K || J == K) return;
  const long long iB = (long long)I * INV_B, jB = (long long)J * INV_B;
  const int r0 = (threadIdx.x >> 4) * 4, c0 = (threadIdx.x & 15) * 4;
  constexpr int H = INV_B / 2;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
#pragma unroll
    for (int t = 0; t < H * INV_B / 2 / INV_T; ++t) {
      const int p = threadIdx.x + t * INV_T, k = h * H + p / (INV_B / 2), c = 2 * (p % (INV_B / 2));
      cp_async16(sW + k * INV_B + c, Wt + (long long)k * np + iB + c);
      cp_async16(sR + k * INV_B + c, Rt + (long long)k * np + jB + c);
    }
    cp_commit();
  }
  double a[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; j += 2)
      *reinterpret_cast<double2*>(&a[i][j]) = *reinterpret_cast<const double2*>(A + (iB + r0 + i) * np + jB + c0 + j);
  cp_wait<1>();
  __syncthreads();
  tile_mac<H, INV_B, true>(sW, sR, a);
  cp_wait<0>();
  __syncthreads();
  tile_mac<H, INV_B, true>(sW + H * INV_B, sR + H * INV_B, a);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; j += 2)
      *reinterpret_cast<double2*>(A + (iB + r0 + i) * np + jB + c0 + j) = *reinterpret_cast<const double2*>(&a[i][j]);
  if (I == K + 1 && J == K + 1) {
    __syncthreads();
    block_invert(a, sW, Pnext, status);
  }
}

__global__ void k_inv_finish(const double* __restrict__ A, int nd, int np, double* __restrict__ Ainv) {
  EDGE_PDL_ENTRY();
  __shared__ double t[32][33];
  // block (by, bx) of 32 x 32 with by >= bx: written in place and mirrored
  const int bx = blockIdx.x, by = blockIdx.y;
  if (bx > by) return;
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  for (int r = y; r < 32; r += 8) {
    const int row = by * 32 + r, col = bx * 32 + x;
    double v = 0.0;
    if (row < nd && col < nd) v = -A[(long long)(row >= col ? row : col) * np + (row >= col ? col : row)];
    t[r][x] = v;
    if (row < nd && col < nd) Ainv[(long long)row * nd + col] = v;
  }
  __syncthreads();
  if (bx == by) return;
  for (int r = y; r < 32; r += 8) {
    const int row = bx * 32 + r, col = by * 32 + x;
    if (row < nd && col < nd) Ainv[(long long)row * nd + col] = t[x][r];
  }
}

int spd_inverse(double* A, int nd, double* Ainv, double* work, int* status, cudaStream_t stream) {
  const int np = inv_padded(nd), nt = np / INV_B;
  double *Rt = work, *Wt = Rt + (long long)INV_B * np, *P0 = Wt + (long long)INV_B * np, *P1 = P0 + INV_B * INV_B;
  constexpr int psmem = 2 * INV_B * INV_LD * 8, usmem = 2 * INV_B * INV_B * 8;
  // on every call: the attributes belong to the current device's context, not to the process
  if (cudaFuncSetAttribute(k_inv_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, psmem) != cudaSuccess ||
      cudaFuncSetAttribute(k_inv_update, cudaFuncAttributeMaxDynamicSharedMemorySize, usmem) != cudaSuccess)
    return 0;
  k_inv_start<<<1, INV_T, 0, stream>>>(A, nd, np, P0, status);
  int n = 1;
  for (int K = 0; K < nt; ++K) {
    k_inv_panel<<<nt, INV_T, psmem, stream>>>(A, np, K, (K & 1) ? P1 : P0, Rt, Wt);
    ++n;
    if (nt > 1) {
      k_inv_update<<<nt * (nt + 1) / 2, INV_T, usmem, stream>>>(A, np, K, Rt, Wt, (K & 1) ? P0 : P1, status);
      ++n;
    }
  }
  const unsigned nb = (unsigned)((nd + 31) / 32);
  k_inv_finish<<<dim3(nb, nb), 256, 0, stream>>>(A, nd, np, Ainv);
  return n + 1;
}

}  // namespace edge
