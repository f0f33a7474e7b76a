"""Performance cases of the SIMP / GMG-PCG framework, through its public Python entry points.

A program that uses the package builds a mesh, a stiffness kernel, a filter, a solver and an
optimiser once and then, iteration after iteration, asks for

  product      K(E) u of the matrix-free FP64 operator           kernel.dot
  filter       the density filter and its transpose              filter.dot, filter.T.dot
  sensitivity  element sensitivities of a displacement           kernel.process_grad
  oc           the optimality-criteria design update             CuTopOpt.update_design
  solve        one GMG-PCG solve from a zero start               CuMultiGrid.solve
  gradient     a differentiable compliance, forward and backward SIMPObjective(...)(rho).backward()
  simp         a whole SIMP iteration, warm-started              CuTopOpt.iterate
  batch        one SIMP iteration of many random 2-D problems    BatchAnalysis

on grids from the 120 x 40 half beam (9,922 DOF) to the 256 x 128 x 128 cantilever (12.8M
DOF), divisible extents and ragged ones (whose multigrid runs on a padded grid).  Elements
are unit squares or cubes with E0 = 1, nu = 0.3, void = 1e-9, penalty 3.

Solves run to rtol 3e-11 (the reference trajectories that designs are compared with use 1e-10,
the gradient checks 1e-12): at the usual 1e-6 two correct solvers differ by what their last
iterations leave.  Solvers are made with their defaults; only the mixed-precision SIMP loop has
its sweeps fixed at one per level and its weight at omega, what the sweep tuner settles on at
12.8M DOF, so that every run times the same algorithm.
"""
import math

import numpy as np
import torch

import edge_to_b200 as eb
from edge_to_b200.batch import BatchAnalysis, build, random_spec

RTOL = 3e-11


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the 120 x 40 half beam's operator: a latency-bound product, as an outer Krylov loop calls it
        {"name": "product 2d 120x40", "kind": "product", "nelx": 120, "nely": 40, "nelz": 0},
        # a ragged 3-D grid: no extent divisible by 4, rows that fill no warp
        {"name": "product 3d 101x51x38", "kind": "product", "nelx": 101, "nely": 51, "nelz": 38},
        # the 12.8M-DOF cantilever's operator: bandwidth
        {"name": "product 3d 256x128x128", "kind": "product", "nelx": 256, "nely": 128, "nelz": 128},
        # design smoothing of the 400 x 200 inverter
        {"name": "filter 2d 400x200", "kind": "filter", "nelx": 400, "nely": 200, "nelz": 0, "rmin": 2.5},
        # the 128 x 64 x 64 differentiation configuration's filter and transpose
        {"name": "filter 3d 128x64x64", "kind": "filter", "nelx": 128, "nely": 64, "nelz": 64, "rmin": 2.0},
        # post-processing of one large analysis
        {"name": "sensitivity 3d 128x64x64", "kind": "sensitivity", "nelx": 128, "nely": 64, "nelz": 64},
        # design updates: the 50-iteration cantilever
        {"name": "oc 3d 64x32x32", "kind": "oc", "nelx": 64, "nely": 32, "nelz": 32, "vf": 0.12},
        # a small FP64 analysis: the half beam, launch latency through and through
        {"name": "solve fp64 2d 120x40", "kind": "solve", "nelx": 120, "nely": 40, "nelz": 0, "levels": 3,
         "precision": "fp64"},
        # a mixed-precision analysis of a grid that the multigrid has to pad
        {"name": "solve mixed 3d 100x50x45", "kind": "solve", "nelx": 100, "nely": 50, "nelz": 45, "levels": 3,
         "precision": "mixed"},
        # forward and backward of a differentiable compliance, FP64
        {"name": "gradient fp64 3d 64x32x32", "kind": "gradient", "nelx": 64, "nely": 32, "nelz": 32, "levels": 4,
         "precision": "fp64", "rmin": 1.5},
        # one SIMP iteration of the 12.8M-DOF cantilever, mixed precision: the headline
        {"name": "simp mixed 3d 256x128x128", "kind": "simp", "nelx": 256, "nely": 128, "nelz": 128, "levels": 5,
         "precision": "mixed", "rmin": 2.0, "vf": 0.1},
        # one SIMP iteration of a batch of random, uneven 2-D problems
        {"name": "batch 2d 24 problems", "kind": "batch", "count": 24, "first": 0, "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any extents for the element-wise calls and the padded
    solves, the grid depths that a program would choose for the solves."""
    kind = rng.choice(["product", "product", "filter", "filter", "sensitivity", "oc", "solve", "solve", "gradient",
                       "simp", "batch"])
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(6, 24), "first": rng.randint(24, 5000),
                "precision": rng.choice(["mixed", "fp64"])}
    if rng.random() < 0.35:
        case = {"kind": kind, "nelx": _log_int(rng, 60, 512), "nely": _log_int(rng, 32, 256), "nelz": 0}
        if kind in ("solve", "gradient", "simp"):
            # slender beams bend so far that the rounding of a true residual nears the tolerance
            case["nelx"] = min(case["nelx"], 400)
            case["nely"] = max(case["nely"], math.ceil(case["nelx"] / 2.5))
    else:
        top = 256 if kind in ("product", "filter", "sensitivity", "oc") else 128
        case = {"kind": kind, "nelx": _log_int(rng, 24, top), "nely": _log_int(rng, 16, top // 2),
                "nelz": _log_int(rng, 16, top // 2)}
    if kind in ("filter", "gradient", "simp"):
        case["rmin"] = round(rng.uniform(1.5, 3.0 if case["nelz"] == 0 else 2.5), 2)
    if kind in ("oc", "simp"):
        case["vf"] = round(rng.uniform(0.1, 0.5), 2)
    if kind in ("solve", "gradient", "simp"):
        case["precision"] = rng.choice(["fp64", "mixed"])
        case["levels"] = rng.randint(3, 4)
    if kind == "simp" or (kind == "gradient" and rng.random() < 0.5):
        # an optimisation loop is laid out on extents that the multigrid coarsens
        m = 2 ** case["levels"]
        for k in ("nelx", "nely", "nelz"):
            if case[k]:
                case[k] = max(m, case[k] // m * m)
    return case


# ------------------------------------------------------------------ what a program holds
def _nel(case):
    return [case["nelx"], case["nely"]] + ([case["nelz"]] if case["nelz"] else [])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(n, gen):
    return torch.rand(n, generator=gen, dtype=torch.float64, device="cuda")


def _randn(n, gen):
    return torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")


def _mesh(case):
    nel = _nel(case)
    cls = eb.CuStructuredMesh2D if len(nel) == 2 else eb.CuStructuredMesh3D
    return cls(*nel, *[float(v) for v in nel], stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))


def _bcs(case):
    """(constrained node ids, per-DOF flags, loaded node ids, force) of the cantilever (3-D: x = 0
    clamped, unit line load on the bottom edge at x = L) or the half beam (2-D: symmetry on
    x = 0, a roller at the bottom right, a unit load at the top left)."""
    nel = _nel(case)
    nx, ny = nel[0] + 1, nel[1] + 1
    if len(nel) == 2:
        left = np.arange(ny) * nx
        return [(left, [[True, False]]), (np.array([nx - 1]), [[False, True]])], np.array([(ny - 1) * nx]), [[0.0, -1.0]]
    nz = nel[2] + 1
    j, k = np.meshgrid(np.arange(ny), np.arange(nz), indexing="ij")
    face = (j * nx * nz + k).ravel()
    edge = nel[0] * nz + np.arange(nz)
    return [(face, [[True, True, True]])], edge, [[0.0, -1.0 / nz, 0.0]]


def _cons_dofs(case):
    nel = _nel(case)
    ids = []
    for nodes, flags in _bcs(case)[0]:
        for c, on in enumerate(flags[0]):
            if on:
                ids.append(nodes * len(nel) + c)
    return np.concatenate(ids)


def _load(case):
    nel = _nel(case)
    f = np.zeros(int(np.prod([v + 1 for v in nel])) * len(nel))
    _, nodes, force = _bcs(case)
    for c, v in enumerate(force[0]):
        f[nodes * len(nel) + c] = v
    return torch.as_tensor(f, device="cuda")


def _filter(case, mesh):
    return (eb.CuStructuredFilter2D if case["nelz"] == 0 else eb.CuStructuredFilter3D)(mesh, case["rmin"])


def _solver(case, mesh, kernel):
    keys = {"tol": RTOL, "maxiter": 2000, "n_level": case["levels"], "precision": case["precision"]}
    if case["kind"] == "simp" and case["precision"] == "mixed":
        keys.update(n_smooth=1, tune_sweeps=False, mixed_omega="max")
    return eb.CuMultiGrid(mesh, kernel, **keys)


def _material(case):
    return eb.SingleMaterial(E=1.0, nu=0.3, void=1e-9, penalty=3.0, volume_fraction=case.get("vf", 0.3))


def _sensitivities(n, rho, gen):
    """Sensitivities of a compliance: negative, spread over several decades, none in voids."""
    return -(rho ** 2) * torch.exp(2.5 * _randn(n, gen))


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed, gen)
    mesh = _mesh(case)
    n_el, n_dof = mesh.n_elements, mesh.n_nodes * mesh.dof
    if kind == "filter":
        flt = _filter(case, mesh)
        rho = _rand(n_el, gen)
        return {"case": case, "filter": flt, "rho": rho, "dr": _sensitivities(n_el, rho, gen)}
    kernel = eb.CuStructuredStiffnessKernel(mesh)
    if kind == "product" or kind == "sensitivity":
        kernel.add_constraints(_cons_dofs(case))
        # a design with solid, grey and void (1e-9) elements
        kernel.set_rho(torch.clamp((1.3 * _rand(n_el, gen) - 0.2).clamp(min=0.0) ** 3, 1e-9, 1.0))
        return {"case": case, "kernel": kernel, "u": _randn(n_dof, gen)}
    solver = None if kind == "oc" else _solver(case, mesh, kernel)
    flt = _filter(case, mesh) if kind in ("gradient", "simp") else None
    mat = _material(case)
    if kind == "solve":
        kernel.add_constraints(_cons_dofs(case))
        kernel.set_rho((0.2 + 0.8 * _rand(n_el, gen)) ** 3)
        return {"case": case, "solver": solver, "f": _load(case)}
    if kind == "gradient":
        kernel.add_constraints(_cons_dofs(case))
        return {"case": case, "kernel": kernel, "solver": solver, "filter": flt, "material": mat, "f": _load(case),
                "rho": (0.2 + 0.8 * _rand(n_el, gen)).requires_grad_(True)}
    opt = eb.CuTopOpt(mesh, mat, kernel, solver, flt, max_iter=1, move=0.2, verbose=False)
    if kind == "oc":
        rho = (2.0 * case["vf"] * _rand(n_el, gen)).clamp(max=1.0)
        return {"case": case, "opt": opt, "rho": rho, "dr": _sensitivities(n_el, rho, gen)}
    # simp: an optimisation that has run its first iterations
    cons, nodes, force = _bcs(case)
    for ids, flags in cons:
        opt.add_BC_nodal(ids, np.array(flags))
    opt.add_F_nodal(nodes, np.array(force))
    rho = case["vf"] * (0.9 + 0.2 * _rand(n_el, gen))
    _, dr, _ = opt.solve_and_process(rho, 0)
    for it in range(2):
        rho, _, dr, _ = opt.iterate(rho, dr, it)
    return {"case": case, "opt": opt, "rho": rho, "dr": dr, "start": solver.last_x0.clone()}


def _prepare_batch(case, seed, gen):
    opts, rhos = [], []
    for i in range(case["count"]):
        spec = random_spec(case["first"] + i)
        opt, rho = build(spec, precision=case["precision"], tol=RTOL, maxiter=2000)
        opt.reuse_sol = False
        opts.append(opt)
        rhos.append(rho * (0.9 + 0.2 * _rand(rho.numel(), gen)))
    batch = BatchAnalysis(opts, threads=1024, team=4, sweeps=(1, 2))
    _, drs, _ = batch.solve_and_process(rhos, 0)
    return {"case": case, "batch": batch, "rhos": rhos, "drs": drs}


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["case"]["kind"]
    if kind == "product":
        return state["kernel"].dot(state["u"])
    if kind == "filter":
        flt = state["filter"]
        return flt.dot(state["rho"]), flt.T.dot(state["dr"])
    if kind == "sensitivity":
        return state["kernel"].process_grad(state["u"])
    if kind == "oc":
        return state["opt"].update_design(state["rho"], state["dr"])
    if kind == "solve":
        x, _ = state["solver"].solve(state["f"], use_last=False)
        return x
    if kind == "gradient":
        rho = state["rho"]
        rho.grad = None
        obj = eb.SIMPObjective(state["kernel"], state["solver"], state["filter"], state["material"], state["f"])
        J = obj(rho)
        J.backward()
        return J.detach(), rho.grad
    if kind == "simp":
        opt = state["opt"]
        opt.solver.last_x0.copy_(state["start"])  # every pass is the same iteration of the loop
        rho, c, dr, _ = opt.iterate(state["rho"], state["dr"], 2)
        return rho, c, dr, opt.solver.last_x0
    batch = state["batch"]
    rhos = batch.update_design(state["rhos"], state["drs"])
    comps, drs, _ = batch.solve_and_process(rhos, 1)
    return torch.cat(rhos), comps, torch.cat([d.reshape(-1) for d in drs])


# ------------------------------------------------------------------ bytes and operations
def work(case):
    """FP64 values that a call reads and writes at least once, and the operations of the
    element transform (about 230 per hex8 element, 50 per Q4) or of the filter taps."""
    kind = case["kind"]
    if kind == "batch":
        el = dof = 0
        for i in range(case["count"]):
            s = random_spec(case["first"] + i)
            el += s["nelx"] * s["nely"]
            dof += 2 * (s["nelx"] + 1) * (s["nely"] + 1)
        return {"bytes": 8.0 * (4 * el + 2 * dof), "flops": 50.0 * el}
    nel = _nel(case)
    el = float(np.prod(nel))
    dof = float(np.prod([v + 1 for v in nel])) * len(nel)
    op = 50.0 if len(nel) == 2 else 230.0
    if kind == "product":
        return {"bytes": 8 * (2 * dof + el), "flops": op * el}
    if kind == "filter":
        return {"bytes": 8 * 4 * el, "flops": 4.0 * el * len(_taps(case)[0])}
    if kind == "sensitivity":
        return {"bytes": 8 * (dof + el), "flops": op * el}
    if kind == "oc":
        return {"bytes": 8 * 3 * el, "flops": 8 * el}
    if kind == "solve":
        return {"bytes": 8 * (2 * dof + el), "flops": op * el}
    if kind == "gradient":
        return {"bytes": 8 * (dof + 2 * el), "flops": 2 * op * el}
    return {"bytes": 8 * (4 * el + 3 * dof), "flops": 2 * op * el}


# ------------------------------------------------------------------ 64-bit values in plain torch
def _element_matrix(dim):
    """Stiffness of the unit square (plane stress) or cube, E = 1, nu = 0.3, 2-point Gauss, with
    the corners in order (0,0) (1,0) (1,1) (0,1) on z = 0, then on z = 1."""
    nu = 0.3
    if dim == 2:
        D = np.array([[1, nu, 0], [nu, 1, 0], [0, 0, (1 - nu) / 2]]) / (1 - nu * nu)
        corners = np.array([[0, 0], [1, 0], [1, 1], [0, 1]], dtype=float)
    else:
        D = np.zeros((6, 6))
        D[:3, :3] = nu
        D[range(3), range(3)] = 1 - nu
        D[range(3, 6), range(3, 6)] = (1 - 2 * nu) / 2
        D /= (1 + nu) * (1 - 2 * nu)
        sq = [[0, 0], [1, 0], [1, 1], [0, 1]]
        corners = np.array([[*p, z] for z in (0, 1) for p in sq], dtype=float)
    pts = (np.array([-1.0, 1.0]) / np.sqrt(3.0) + 1) / 2
    K = np.zeros((len(corners) * dim,) * 2)
    for q in np.stack(np.meshgrid(*[pts] * dim, indexing="ij"), -1).reshape(-1, dim):
        N1 = np.where(corners == 1, q, 1 - q)
        g = np.stack([np.prod(np.delete(N1, a, 1), 1) * np.where(corners[:, a] == 1, 1.0, -1.0) for a in range(dim)], 1)
        B = np.zeros((D.shape[0], K.shape[0]))
        for a in range(dim):
            B[a, a::dim] = g[:, a]
        for row, (a, b) in enumerate([(0, 1)] if dim == 2 else [(0, 1), (1, 2), (0, 2)]):
            B[dim + row, a::dim] = g[:, b]
            B[dim + row, b::dim] = g[:, a]
        K += B.T @ D @ B / 2 ** dim
    return torch.as_tensor(K, device="cuda")


def _element_dofs(nel):
    """DOFs of every element (n_el x corners * dim), elements i outermost, then j, then k."""
    dim = len(nel)
    ax = [torch.arange(v, device="cuda") for v in nel]
    nx = nel[0] + 1
    if dim == 2:
        base = ax[1][None, :] * nx + ax[0][:, None]
        off = [0, 1, nx + 1, nx]
    else:
        nz = nel[2] + 1
        base = (ax[1][None, :, None] * nx + ax[0][:, None, None]) * nz + ax[2][None, None, :]
        off = [0, nz, nz + nx * nz, nx * nz]
        off = off + [o + 1 for o in off]
    nodes = base.reshape(-1, 1) + torch.tensor(off, device="cuda")[None]
    return (nodes[:, :, None] * dim + torch.arange(dim, device="cuda")).reshape(nodes.shape[0], -1)


def _taps(case):
    dim = 2 if case["nelz"] == 0 else 3
    n = math.ceil(case["rmin"])
    offs = np.stack(np.meshgrid(*[np.arange(-n, n + 1)] * dim, indexing="ij"), -1).reshape(-1, dim)
    w = 1 - np.linalg.norm(offs, axis=1) / case["rmin"]
    return offs[w > 0], w[w > 0]


def _shifted(x, off):
    """x shifted by off with zeros from outside: y[e] = x[e + off]."""
    y = torch.zeros_like(x)
    dst, src = [], []
    for o, n in zip(off, x.shape):
        o = int(o)
        if abs(o) >= n:
            return y
        dst.append(slice(max(0, -o), n - max(0, o)))
        src.append(slice(max(0, o), n - max(0, -o)))
    y[tuple(dst)] = x[tuple(src)]
    return y


def _exact_product(case, seed):
    nel = _nel(case)
    gen = _gen(seed)
    n_el = int(np.prod(nel))
    n_dof = int(np.prod([v + 1 for v in nel])) * len(nel)
    E = torch.clamp((1.3 * _rand(n_el, gen) - 0.2).clamp(min=0.0) ** 3, 1e-9, 1.0)
    u = _randn(n_dof, gen)
    K0, dofs = _element_matrix(len(nel)), _element_dofs(nel)
    if case["kind"] == "sensitivity":
        out = torch.empty(n_el, dtype=torch.float64, device="cuda")
        for s in range(0, n_el, 1 << 18):
            ue = u[dofs[s:s + (1 << 18)]]
            out[s:s + (1 << 18)] = -((ue @ K0) * ue).sum(1)
        return out
    cons = torch.as_tensor(_cons_dofs(case), device="cuda")
    v = u.clone()
    v[cons] = 0.0
    out = torch.zeros_like(u)
    for s in range(0, n_el, 1 << 18):
        d = dofs[s:s + (1 << 18)]
        out.index_add_(0, d.reshape(-1), (E[s:s + (1 << 18), None] * (v[d] @ K0)).reshape(-1))
    out[cons] = u[cons]
    return out


def _exact_filter(case, seed):
    nel = _nel(case)
    gen = _gen(seed)
    n_el = int(np.prod(nel))
    rho = _rand(n_el, gen)
    dr = _sensitivities(n_el, rho, gen).reshape(nel)
    rho = rho.reshape(nel)
    offs, w = _taps(case)
    norm, fwd = torch.zeros_like(rho), torch.zeros_like(rho)
    one = torch.ones_like(rho)
    for o, wk in zip(offs, w):
        norm += wk * _shifted(one, o)
        fwd += wk * _shifted(rho, o)
    back = torch.zeros_like(rho)
    for o, wk in zip(offs, w):
        back += wk * _shifted(dr / norm, o)
    return (fwd / norm).reshape(-1), back.reshape(-1)


def _exact_oc(case, seed):
    gen = _gen(seed)
    n_el = int(np.prod(_nel(case)))
    rho = (2.0 * case["vf"] * _rand(n_el, gen)).clamp(max=1.0)
    dr = _sensitivities(n_el, rho, gen)
    ocp = (rho * torch.sqrt((-dr).clamp(min=0.0))).clamp(min=1e-12)
    lo, hi = (rho - 0.2).clamp(0.0, 1.0), (rho + 0.2).clamp(0.0, 1.0)
    l1, l2 = 1e-9, 1e9
    new = rho
    while (l2 - l1) / (l2 + l1) > 1e-4:
        mid = 0.5 * (l1 + l2)
        new = torch.maximum(lo, torch.minimum(hi, ocp / mid))
        if float(new.sum()) / n_el <= case["vf"]:
            l2 = mid
        else:
            l1 = mid
    return new


def _exact_solve(case, seed):
    """The assembled system solved densely (small grids only)."""
    nel = _nel(case)
    n_dof = int(np.prod([v + 1 for v in nel])) * len(nel)
    if n_dof > 16000:
        return None
    E = (0.2 + 0.8 * _rand(int(np.prod(nel)), _gen(seed))) ** 3
    K0, dofs = _element_matrix(len(nel)), _element_dofs(nel)
    m = dofs.shape[1]
    K = torch.zeros(n_dof * n_dof, dtype=torch.float64, device="cuda")
    K.index_add_(0, (dofs[:, :, None] * n_dof + dofs[:, None, :]).reshape(-1), (E[:, None, None] * K0).reshape(-1))
    K = K.reshape(n_dof, n_dof)
    free = torch.ones(n_dof, dtype=torch.bool, device="cuda")
    free[torch.as_tensor(_cons_dofs(case), device="cuda")] = False
    ix = torch.nonzero(free).reshape(-1)
    f = _load(case)
    A = K[ix][:, ix]
    L = torch.linalg.cholesky(A)
    b = f[ix, None]
    x = torch.cholesky_solve(b, L)
    for _ in range(2):  # iterative refinement
        x = x + torch.cholesky_solve(b - A @ x, L)
    out = torch.zeros_like(f)
    out[ix] = x.reshape(-1)
    return out


def exact(case, seed):
    """The same outputs in plain 64-bit torch; None for solves too large to assemble densely and for
    the calls that contain one."""
    kind = case["kind"]
    if kind in ("product", "sensitivity"):
        return _exact_product(case, seed)
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind == "oc":
        return _exact_oc(case, seed)
    if kind == "solve":
        return _exact_solve(case, seed)
    return None
