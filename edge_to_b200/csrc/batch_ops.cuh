// Passes of a team of blocks (one block, or a thread block cluster) over one level of a 2-D problem: the
// fine operator, stencils, transfers, smoothing, the coarsest product and team-wide sums, for the batched
// solve (batch.cu) and the one-launch cycle of the per-problem solver (vtail.cu).
#pragma once
#include "batch.cuh"

#include <cooperative_groups.h>

namespace edge {

constexpr int BATCH_COARSE_SMEM = 1024;  // coarsest right-hand sides up to this size are staged in shared memory

// The blocks that solve one problem together.
template <int C> struct Team {
  static EDGE_D unsigned rank() {
    if constexpr (C == 1) return 0;
    else return cooperative_groups::this_cluster().block_rank();
  }
  static EDGE_D int first() { return (int)(rank() * blockDim.x + threadIdx.x); }
  static EDGE_D int stride() { return C * (int)blockDim.x; }
  static EDGE_D void sync() {
    if constexpr (C == 1) __syncthreads();
    else cooperative_groups::this_cluster().sync();
  }
};

// Team-wide FP64 sums, returned to every thread; the sum is also a team barrier.  Team sizes are chosen
// by what else is solved beside a problem, so the order of a sum must not follow them: the terms are
// those of TEAM_MAX virtual blocks whatever the team's size C (term k belongs to thread k mod BT of
// virtual block (k / BT) mod TEAM_MAX), a block of the team adds up its TEAM_MAX / C virtual blocks one
// after the other, and the TEAM_MAX block sums are added in their order.  A thread handles the terms that
// a plain stride over the team would give it.
//
// pass(first, step, acc) adds the terms first, first + step, ... to acc.  sh: TeamSum<C>::SH doubles of
// shared memory; ph alternates between the two halves of the block sums from sum to sum (alike in every
// thread).  Each block writes its block sums into every block's shared memory, so that after one
// cluster barrier all threads read locally.
constexpr int TEAM_MAX = 16;
template <int C> struct TeamSum {
  static constexpr int PER = TEAM_MAX / C;      // virtual blocks of a block
  static constexpr int SH = PER * 32 + 2 * TEAM_MAX;  // their warps' sums, the block sums
  template <class Pass> static EDGE_D double run(Pass&& pass, double* sh, int& ph) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5, BT = blockDim.x;
    const int rank = (int)Team<C>::rank();
    double* half = sh + PER * 32 + ph * TEAM_MAX;
    for (int q = 0; q < PER; ++q) {
      double acc = 0.0;
      pass((rank + q * C) * BT + (int)threadIdx.x, TEAM_MAX * BT, acc);
      acc = warp_sum(acc);
      if (lane == 0) sh[q * 32 + wid] = acc;  // read last before the previous sum's team barrier
    }
    __syncthreads();
    for (int q = wid; q < PER; q += nw) {
      const double r = warp_sum(lane < nw ? sh[q * 32 + lane] : 0.0);
      if constexpr (C == 1) {
        if (lane == 0) half[q] = r;
      } else {
        if (lane < C) *cooperative_groups::this_cluster().map_shared_rank(half + rank + q * C, lane) = r;
      }
    }
    Team<C>::sync();
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < TEAM_MAX; ++k) t += half[k];
    ph ^= 1;  // this half is written again two sums from now, behind the next sum's barrier
    return t;
  }
};

// Fine-level operator of a 2-D problem, one pass of the block over the level's nodes: at
// node (i, j), A u from the 3 x 3 neighbourhood (constrained components of u read as zero)
// and the four surrounding elements' E with the dense element matrix sK (corner-bit order,
// shared memory), in the order of k_fine2_dense; identity rows on constrained DOFs.
// epi(s, own, Au) finishes node slot s (own: the node's raw input values).  Every load of a
// node is unconditional (a neighbour or element outside the grid reads the node's own slot
// and is replaced by zero), so a thread's loads are in flight together: each pass is a few
// round trips to L2 per node, not one per neighbour.
// uin(slot, component): the input's values.  The form of the FP64 product, and of any element matrix
// without the box structure.  The product keeps it where the preconditioner marches in the transform
// domain (below): on slender problems the solution follows the last bits of the Krylov operator (in 8
// problems drawn at random the designs moved by 5e-9 of their size with the transform, by 5e-12 with this
// form), and marching with the full matrix in this order of sums spills at 1024 threads (354 ms a solve of
// those 8 problems, 171 with this form).
template <int C, typename T, typename TE, class UIn, class F>
EDGE_D void b_fine2(const Geo& g, UIn uin, const TE* E, const uint8_t* mask, const T* sK, F&& epi,
                    int first = Team<C>::first(), int step = Team<C>::stride()) {
  const int nn = g.nx * g.ny;
  for (int t = first; t < nn; t += step) {
    const int i = t % g.nx, j = t / g.nx;
    const long long s = g.slot2(i, j);
    T U[3][3][2];
#pragma unroll
    for (int dy = 0; dy < 3; ++dy)
#pragma unroll
      for (int dx = 0; dx < 3; ++dx) {
        const int ii = i + dx - 1, jj = j + dy - 1;
        const bool in = ii >= 0 && ii < g.nx && jj >= 0 && jj < g.ny;
        const long long ss = in ? s + (long long)(dy - 1) * g.pz + (dx - 1) : s;
        const uint8_t mr = __ldg(mask + ss);
        const uint8_t m = in ? mr : (uint8_t)3;
        const T a0 = uin(ss, 0), a1 = uin(ss, 1);
        U[dy][dx][0] = (m & 1) ? T(0) : a0;
        U[dy][dx][1] = (m & 2) ? T(0) : a1;
      }
    T Au[2] = {T(0), T(0)};
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int ax = a & 1, ay = a >> 1;
      const int li = i - ax, lj = j - ay;
      const bool ev = li >= 0 && lj >= 0 && li < g.nx - 1 && lj < g.ny - 1;
      const TE Ev = __ldg(E + (ev ? g.slot2(li, lj) : s));
      const T Ee = ev ? Conv<T>::from(Ev) : T(0);
      T r[2] = {T(0), T(0)};
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int bx = b & 1, by = b >> 1;
#pragma unroll
        for (int dd = 0; dd < 2; ++dd) {
          const T ub = U[by - ay + 1][bx - ax + 1][dd];
#pragma unroll
          for (int c = 0; c < 2; ++c) r[c] += sK[(a * 2 + c) * 8 + b * 2 + dd] * ub;
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) Au[c] += Ee * r[c];
    }
    const uint8_t m = __ldg(mask + s);
    T own[2] = {uin(s, 0), uin(s, 1)};
    Au[0] = (m & 1) ? own[0] : Au[0];
    Au[1] = (m & 2) ? own[1] : Au[1];
    epi(s, own, Au);
  }
}

// The same operator marching along y, for element matrices with the box structure: a warp owns 32 element
// columns (30 nodes besides its halo lanes) and a strip of rows, a lane one element per row.  A row
// costs a lane one node (value, mask) and one E; its right neighbour's node and its left neighbour's
// contributions come by shuffle, the lower row of nodes and the contributions to the upper one stay in
// registers, and the element works in the transform domain (10 coefficients, 48 operations) where
// the node-wise form loads nine nodes and four E and multiplies four 8 x 2 blocks.  The next row's
// loads are issued a row ahead.  A sweep's pass takes
// about two thirds of the node-wise pass's time.
// uin(i, j, s, v): the input at node (i, j), slot s.
template <int C, typename T, typename TE, class UIn, class F>
EDGE_D void b_fine2_march(const Geo& g, UIn uin, const TE* E, const uint8_t* mask, const KHat2<T>& K, F&& epi) {
  const int lane = threadIdx.x & 31, wid = Team<C>::first() >> 5, nwarp = Team<C>::stride() >> 5;
  const int ct = (g.nx + 29) / 30;                         // column tiles of 30 nodes
  const int want = nwarp / ct > 0 ? nwarp / ct : 1;        // strips per column tile
  const int rows = (g.ny + want - 1) / want, strips = (g.ny + rows - 1) / rows;
  const T k10 = K.dg[0][1], k20 = K.dg[0][2], k30 = K.dg[0][3], k11 = K.dg[1][1], k21 = K.dg[1][2], k31 = K.dg[1][3];
  const T o01 = K.of[0][1][1], o02 = K.of[0][1][2], o11 = K.of[1][0][1], o12 = K.of[1][0][2];
  for (int t = wid; t < ct * strips; t += nwarp) {
    const int cx = t % ct, y0 = (t / ct) * rows, y1 = min(y0 + rows, g.ny);
    const int i = cx * 30 - 1 + lane;  // this lane's node and element column
    const bool ni = i >= 0 && i < g.nx;
    const int ic = ni ? i : 0;
    struct Row {
      T raw[2], E;
      unsigned m;
    };
    auto fetch = [&](int j) {  // node (i, j) and the E of element (i, j); clamped loads, zeroed after
      Row r;
      const int jc = min(max(j, 0), g.ny - 1);
      const long long s = g.slot2(ic, jc);
      const bool in = ni && j >= 0 && j < g.ny;
      uin(ic, jc, s, r.raw);
      const unsigned m = __ldg(mask + s);
      const T e = Conv<T>::from(__ldg(E + s));
      r.m = in ? m : 3u;
      r.E = in ? e : T(0);  // slots past the last element hold zero
      return r;
    };
    Row lo = fetch(y0 - 1), hi = fetch(y0);
    T ul[2], cl[2] = {T(0), T(0)}, cr[2] = {T(0), T(0)};  // masked lower node; contributions carried upwards
    T ulr[2];                                              // the right neighbour's lower node
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      ul[c] = ((lo.m >> c) & 1) ? T(0) : lo.raw[c];
      ulr[c] = __shfl_down_sync(0xffffffffu, ul[c], 1);
    }
    for (int j = y0 - 1; j < y1; ++j) {  // element row j: nodes j (lo) and j + 1 (hi)
      const Row nx = fetch(j + 2);
      T uh[2], uhr[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uh[c] = ((hi.m >> c) & 1) ? T(0) : hi.raw[c];
        uhr[c] = __shfl_down_sync(0xffffffffu, uh[c], 1);
      }
      // transform of the corners b = bx + 2 by, h = hx + 2 hy
      T q[2][4], v[2][4];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const T sl = ul[c] + ulr[c], dl = ul[c] - ulr[c], su = uh[c] + uhr[c], du = uh[c] - uhr[c];
        q[c][1] = (dl + du) * lo.E;
        q[c][2] = (sl - su) * lo.E;
        q[c][3] = (dl - du) * lo.E;
      }
      v[0][1] = k10 * q[0][1] + o01 * q[1][2];
      v[0][2] = k20 * q[0][2] + o02 * q[1][1];
      v[0][3] = k30 * q[0][3];
      v[1][1] = k11 * q[1][1] + o11 * q[0][2];
      v[1][2] = k21 * q[1][2] + o12 * q[0][1];
      v[1][3] = k31 * q[1][3];
      T Au[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        // contributions to corners (0,0) (1,0) (0,1) (1,1); h = 0 vanishes
        const T a = v[c][1] + v[c][2], b = v[c][2] - v[c][1], d = v[c][1] - v[c][2];
        const T f00 = a + v[c][3], f10 = b - v[c][3], f01 = d - v[c][3], f11 = v[c][3] - a;
        // node (i, j): this element's corner (0,0), the left element's (1,0), and the row below's
        // (0,1) and (1,1) carried from the previous row
        Au[c] = f00 + cl[c] + __shfl_up_sync(0xffffffffu, f10 + cr[c], 1);
        cl[c] = f01;
        cr[c] = f11;
      }
      if (j >= y0 && lane >= 1 && lane <= 30 && ni) {
        const long long s = g.slot2(i, j);
#pragma unroll
        for (int c = 0; c < 2; ++c)
          if ((lo.m >> c) & 1) Au[c] = lo.raw[c];
        epi(s, lo.raw, Au);
      }
      lo = hi;
      hi = nx;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        ul[c] = uh[c];
        ulr[c] = uhr[c];
      }
    }
  }
}
// The element matrix of a problem in shared memory: dense, and its transform when it has the box
// structure (else null).
template <typename T> struct FineK {
  const T* dense;
  const KHat2<T>* k2;
};
// Input values of the fine operator: an array of the level.
template <typename T> struct NodeIn {
  const T* u;
  long long n;
  EDGE_D void operator()(int, int, long long s, T v[2]) const {
    v[0] = u[s];
    v[1] = u[n + s];
  }
};
// ... or the interpolation of a coarse array (b_prolong2's values: the mean over a node's parents; an
// even coordinate counts its one parent twice).
template <typename T> struct ProlongIn {
  Geo gc;
  const T* e;
  EDGE_D void operator()(int i, int j, long long, T v[2]) const {
    v[0] = v[1] = T(0);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int ci = min((i + a) >> 1, gc.nx - 1), cj = min((j + b) >> 1, gc.ny - 1);
        const T iw = inv_bnd_total2<T>(is_bnd(ci, gc.nx) + is_bnd(cj, gc.ny));
        const long long sc = gc.slot2(ci, cj);
        v[0] += e[sc] * iw;
        v[1] += e[gc.n + sc] * iw;
      }
    v[0] *= T(0.25);
    v[1] *= T(0.25);
  }
};
// The fine-level operator in either form; uin(i, j, s, v) as above.
template <int C, typename T, typename TE, class UIn, class F>
EDGE_D void b_fine2_op(const Geo& g, UIn uin, const TE* E, const uint8_t* mask, const FineK<T>& K, F&& epi) {
  if (K.k2) {
    b_fine2_march<C, T, TE>(g, uin, E, mask, *K.k2, epi);
  } else {
    const T* sK = K.dense;
    b_fine2<C, T, TE>(g, [&](long long ss, int c) {
      T v[2];
      uin((int)(ss % g.pz), (int)(ss / g.pz), ss, v);
      return v[c];
    }, E, mask, sK, epi);
  }
}

// Symmetric 2-D stencil (levels >= 1), one pass of the block over the level's nodes, the
// sums of k_st2_apply in its order (a neighbour outside the grid reads the node's own slots
// and contributes zero, so no load is conditional).
template <int C, typename T, typename TS, class F>
EDGE_D void b_st2(const Geo& g, const T* u, const TS* S, F&& epi) {
  const long long n = g.n;
  const int nn = g.nx * g.ny;
  for (int t = Team<C>::first(); t < nn; t += Team<C>::stride()) {
    const int i = t % g.nx, j = t / g.nx;
    const long long s = g.slot2(i, j);
    const T u0 = u[s], u1 = u[n + s];
    const T c00 = Conv<T>::from(__ldg(S + s)), c01 = Conv<T>::from(__ldg(S + n + s)),
            c11 = Conv<T>::from(__ldg(S + 2 * n + s));
    T Au[2];
    Au[0] = c00 * u0 + c01 * u1;
    Au[1] = c01 * u0 + c11 * u1;
#pragma unroll
    for (int nb = 5; nb < 9; ++nb) {
      const int dx = nb % 3 - 1, dy = nb / 3 - 1;
      const long long off = (long long)dy * g.pz + dx;
      const TS* Sb = S + (long long)(3 + (nb - 5) * 4) * n;
      {
        const bool in = i + dx >= 0 && i + dx < g.nx && j + dy >= 0 && j + dy < g.ny;
        const long long sn = in ? s + off : s;
        const T v0 = in ? u[sn] : T(0), v1 = in ? u[n + sn] : T(0);
        Au[0] += Conv<T>::from(__ldg(Sb + s)) * v0 + Conv<T>::from(__ldg(Sb + n + s)) * v1;
        Au[1] += Conv<T>::from(__ldg(Sb + 2 * n + s)) * v0 + Conv<T>::from(__ldg(Sb + 3 * n + s)) * v1;
      }
      {
        const bool in = i - dx >= 0 && i - dx < g.nx && j - dy >= 0 && j - dy < g.ny;
        const long long sm = in ? s - off : s;
        const T v0 = in ? u[sm] : T(0), v1 = in ? u[n + sm] : T(0);
        Au[0] += Conv<T>::from(__ldg(Sb + sm)) * v0 + Conv<T>::from(__ldg(Sb + 2 * n + sm)) * v1;
        Au[1] += Conv<T>::from(__ldg(Sb + n + sm)) * v0 + Conv<T>::from(__ldg(Sb + 3 * n + sm)) * v1;
      }
    }
    T own[2] = {u0, u1};
    epi(s, own, Au);
  }
}

// Full-weighting restriction to the coarse nodes (k_restrict2's sums); with x given, also the coarse
// level's first sweep from zero, x = w Dinv out.
template <int C, typename T>
EDGE_D void b_restrict2(const Geo& gf, const Geo& gc, const T* in, T* out, const T* dinv, T w, T* x) {
  const int nc = gc.nx * gc.ny;
  for (int t = Team<C>::first(); t < nc; t += Team<C>::stride()) {
    const int I = t % gc.nx, J = t / gc.nx;
    const T iw = inv_bnd_total2<T>(is_bnd(I, gc.nx) + is_bnd(J, gc.ny));
    T v[2] = {0, 0};
#pragma unroll
    for (int di = -1; di <= 1; ++di) {
      const int fi = 2 * I + di;
#pragma unroll
      for (int dj = -1; dj <= 1; ++dj) {  // unconditional loads: outside the grid the centre, weight 0
        const int fj = 2 * J + dj;
        const bool ok = fi >= 0 && fi < gf.nx && fj >= 0 && fj < gf.ny;
        const T wt = ok ? (T)(0.25 * (2 - (di != 0)) * (2 - (dj != 0))) : T(0);
        const long long sf = gf.slot2(ok ? fi : 2 * I, ok ? fj : 2 * J);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const T a = in[c * gf.n + sf];
          v[c] += ok ? wt * a : T(0);
        }
      }
    }
    const long long sc = gc.slot2(I, J);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const T o = v[c] * iw;
      out[c * gc.n + sc] = o;
      if (x) x[c * gc.n + sc] = w * __ldg(dinv + c * gc.n + sc) * o;
    }
  }
}

// Interpolation to the fine nodes (k_prolong2's sums).
template <int C, typename T>
EDGE_D void b_prolong2(const Geo& gf, const Geo& gc, const T* in, T* out) {
  const int nf = gf.nx * gf.ny;
  for (int t = Team<C>::first(); t < nf; t += Team<C>::stride()) {
    const int i = t % gf.nx, j = t / gf.nx;
    T v[2] = {0, 0};
    int cnt = 0;
    for (int ci = i / 2; ci <= i / 2 + (i & 1); ++ci) {
      if (ci >= gc.nx) continue;
      for (int cj = j / 2; cj <= j / 2 + (j & 1); ++cj) {
        if (cj >= gc.ny) continue;
        const T iw = inv_bnd_total2<T>(is_bnd(ci, gc.nx) + is_bnd(cj, gc.ny));
        const long long sc = gc.slot2(ci, cj);
        for (int c = 0; c < 2; ++c) v[c] += in[c * gc.n + sc] * iw;
        ++cnt;
      }
    }
    const T ic = cnt ? T(1) / T(cnt) : T(0);
    const long long sf = gf.slot2(i, j);
    for (int c = 0; c < 2; ++c) out[c * gf.n + sf] = v[c] * ic;
  }
}

// x = Ainv b on the coarsest level (dense order: DOF c of node j * nx + i), one warp per row;
// every block of the team stages b (written before the team's last barrier) for its rows.
template <int C, typename T>
EDGE_D void b_coarse2(const Geo& g, const double* Ainv, int nd, const T* b, T* x, double* sb) {
  auto slot_of = [&](int dn) -> long long {
    const int node = dn >> 1;
    return (long long)(dn & 1) * g.n + g.slot2(node % g.nx, node / g.nx);
  };
  const bool staged = nd <= BATCH_COARSE_SMEM;
  if (staged) {
    for (int c = threadIdx.x; c < nd; c += blockDim.x) sb[c] = (double)b[slot_of(c)];
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, nw = Team<C>::stride() >> 5;
  for (int row = Team<C>::first() >> 5; row < nd; row += nw) {
    const double* a = Ainv + (long long)row * nd;
    double acc = 0.0;
    for (int c = lane; c < nd; c += 32) acc += __ldg(a + c) * (staged ? sb[c] : (double)b[slot_of(c)]);
    acc = warp_sum(acc);
    if (lane == 0) x[slot_of(row)] = Conv<T>::from(acc);
  }
}

template <int C, typename TA, typename TB>
EDGE_D double b_dot(long long nv, const TA* a, const TB* b, double* sh, int& ph) {
  return TeamSum<C>::run([&](int first, int step, double& acc) {
    for (long long q = first; q < nv; q += step) acc += (double)a[q] * (double)b[q];
  }, sh, ph);
}

// One application of level l's operator (fine: the element operator in TV; coarser: the
// stencil in TS, arithmetic in TV).
template <int C, typename TV, typename TS, class F>
EDGE_D void b_level_op(const BatchDesc& d, int l, const TV* u, const FineK<TV>& sK, F&& epi) {
  if (l == 0)
    b_fine2_op<C, TV, TV>(d.lv[0].g, NodeIn<TV>{u, d.lv[0].g.n}, (const TV*)d.ET, d.mask, sK, epi);
  else
    b_st2<C, TV, TS>(d.lv[l].g, u, (const TS*)d.lv[l].S, epi);
}

// Damped-Jacobi pieces with level l's inverse diagonal (type TD); the level's right-hand side
// b has type TB (level 0: the FP64 PCG residual, read in the V-cycle's type).  down: x = w
// Dinv b (k_jacobi0), ns - 1 more sweeps, r = b - A x; with one sweep on level 0 the two are
// one pass (the operator's input w Dinv b computed where it is read, x never stored: fused0).
// up (after the interpolation into e1): ns - 1 sweeps on the correction, then
// out = xb + (e + w Dinv (r - A e)) with xb the down pass's x (recomputed as w Dinv b when
// fused0).
template <int C, typename TV, typename TS, typename TD, typename TB>
EDGE_D void b_smooth_level(const BatchDesc& d, int l, const FineK<TV>& sK, TV w, const TB* b, const TV* xb, TV*& x, TV*& y,
                           TV*& e1, TV*& e2, TV* r, TV* out, bool down, bool fused0, bool pre_done) {
  using TM = Team<C>;
  const BatchLevel& Lv = d.lv[l];
  const Geo& g = Lv.g;
  const long long n = g.n, nv = 2 * n;
  const TD* D = (const TD*)Lv.dinv;
  const int ns = d.sweeps[l];
  auto bv = [&](long long q) { return Conv<TV>::from(b[q]); };
  auto wdb = [&](long long q) { return w * Conv<TV>::from(__ldg(D + q)) * bv(q); };
  auto sweep = [&](const TV* bb, const TV* in, TV* o) {
    b_level_op<C, TV, TS>(d, l, in, sK, [&](long long s, const TV* own, const TV* Au) {
      for (int c = 0; c < 2; ++c) {
        const long long q = c * n + s;
        o[q] = own[c] + w * Conv<TV>::from(__ldg(D + q)) * (bb[q] - Au[c]);
      }
    });
    TM::sync();
  };
  auto sweep_b = [&](const TV* in, TV* o) {  // a sweep on the down pass (right-hand side b)
    b_level_op<C, TV, TS>(d, l, in, sK, [&](long long s, const TV* own, const TV* Au) {
      for (int c = 0; c < 2; ++c) {
        const long long q = c * n + s;
        o[q] = own[c] + w * Conv<TV>::from(__ldg(D + q)) * (bv(q) - Au[c]);
      }
    });
    TM::sync();
  };
  if (down) {
    if (fused0) {
      b_fine2_op<C, TV, TV>(g, [&](int, int, long long ss, TV* v) {
        v[0] = wdb(ss);
        v[1] = wdb(n + ss);
      }, (const TV*)d.ET, d.mask, sK, [&](long long s, const TV* own, const TV* Au) {
                           for (int c = 0; c < 2; ++c) r[c * n + s] = bv(c * n + s) - Au[c];
                         });
      TM::sync();
      return;
    }
    if (ns >= 1) {
      if (!pre_done) {
        for (long long q = TM::first(); q < nv; q += TM::stride()) x[q] = wdb(q);
        TM::sync();
      }
      for (int s = 1; s < ns; ++s) {
        sweep_b(x, y);
        TV* t = x;
        x = y;
        y = t;
      }
    } else {
      for (long long q = TM::first(); q < nv; q += TM::stride()) x[q] = TV(0);
      TM::sync();
    }
    b_level_op<C, TV, TS>(d, l, x, sK, [&](long long s, const TV* own, const TV* Au) {
      for (int c = 0; c < 2; ++c) r[c * n + s] = bv(c * n + s) - Au[c];
    });
    TM::sync();
  } else {
    for (int s = 0; s + 1 < ns; ++s) {
      sweep(r, e1, e2);
      TV* t = e1;
      e1 = e2;
      e2 = t;
    }
    auto xbase = [&](long long q) { return fused0 ? wdb(q) : xb[q]; };
    if (ns >= 1) {
      auto last = [&](long long s, const TV* own, const TV* Au) {
        for (int c = 0; c < 2; ++c) {
          const long long q = c * n + s;
          const TV e = own[c] + w * Conv<TV>::from(__ldg(D + q)) * (r[q] - Au[c]);
          out[q] = xbase(q) + e;
        }
      };
      if (fused0)  // the correction is interpolated where it is read (b_vcycle skips the pass)
        b_fine2_op<C, TV, TV>(g, ProlongIn<TV>{d.lv[1].g, (const TV*)d.lv[1].res}, (const TV*)d.ET, d.mask, sK, last);
      else
        b_level_op<C, TV, TS>(d, l, e1, sK, last);
    } else {
      for (long long q = TM::first(); q < nv; q += TM::stride()) out[q] = Conv<TV>::from((double)xb[q] + (double)e1[q]);
    }
    TM::sync();
  }
}

// Levels [l0, l1) of a V-cycle downwards (smoothing, residual, restriction with the next level's first
// sweep; pre_done: level l0's own first sweep was done that way) and upwards.  xcur: the levels' iterates.
template <int C, typename TV, typename TD0, typename TS>
EDGE_D void b_down(const BatchDesc& d, const FineK<TV>& sK, double omega, int l0, int l1, TV** xcur) {
  for (int l = l0; l < l1; ++l) {
    const BatchLevel& Lv = d.lv[l];
    TV* x = (TV*)Lv.xa;
    TV* y = (TV*)Lv.xb;
    TV* e1 = nullptr;
    TV* e2 = nullptr;
    const TV w = Conv<TV>::from(omega * d.wscale[l]);
    if (l == 0)
      b_smooth_level<C, TV, TS, TD0, double>(d, l, sK, w, d.r64, nullptr, x, y, e1, e2, (TV*)Lv.r, nullptr, true,
                                              d.sweeps[0] == 1, false);
    else
      b_smooth_level<C, TV, TS, TV, TV>(d, l, sK, w, (const TV*)Lv.b, nullptr, x, y, e1, e2, (TV*)Lv.r, nullptr,
                                        true, false, d.sweeps[l] >= 1);
    xcur[l] = x;
    const BatchLevel& Lc = d.lv[l + 1];
    const bool j0 = l + 1 < d.n_level && d.sweeps[l + 1] >= 1;
    b_restrict2<C, TV>(Lv.g, Lc.g, (const TV*)Lv.r, (TV*)Lc.b, (const TV*)Lc.dinv,
                       Conv<TV>::from(omega * d.wscale[l + 1]), j0 ? (TV*)Lc.xa : nullptr);
    Team<C>::sync();
  }
}
template <int C, typename TV, typename TD0, typename TS>
EDGE_D void b_up(const BatchDesc& d, const FineK<TV>& sK, double omega, int l0, int l1, TV** xcur) {
  for (int l = l1 - 1; l >= l0; --l) {
    const BatchLevel& Lv = d.lv[l];
    const bool fused0 = l == 0 && d.sweeps[0] == 1;
    TV* e1 = (TV*)Lv.ea;
    TV* e2 = (TV*)Lv.eb;
    TV* x = nullptr;
    TV* y = nullptr;
    if (!fused0) {
      b_prolong2<C, TV>(Lv.g, d.lv[l + 1].g, (const TV*)d.lv[l + 1].res, e1);
      Team<C>::sync();
    }
    const TV w = Conv<TV>::from(omega * d.wscale[l]);
    if (l == 0)
      b_smooth_level<C, TV, TS, TD0, double>(d, l, sK, w, d.r64, xcur[l], x, y, e1, e2, (TV*)Lv.r, (TV*)Lv.res,
                                              false, fused0, false);
    else
      b_smooth_level<C, TV, TS, TV, TV>(d, l, sK, w, (const TV*)Lv.b, xcur[l], x, y, e1, e2, (TV*)Lv.r,
                                        (TV*)Lv.res, false, false, false);
  }
}

}  // namespace edge
