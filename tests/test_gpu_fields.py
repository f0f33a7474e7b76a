"""Element-wise passes on user-layout arrays (csrc/fields.cu) against the CPU oracle, at the
sizes where their tiles and blocks end."""
import ctypes

import numpy as np
import pytest

from oracle import ops, topopt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 148 * 512 - 1, 148 * 512 + 1, 1048576])
@pytest.mark.parametrize("vf", [0.05, 0.5, 0.999])
def test_oc_update_equals_sequential_bisection(n, vf):
    """Same multiplier, step count and design as the oracle's step-by-step bisection; the sums differ
    in their order only (n terms of at most 1: 1e-16 sqrt(n), far from any decision)."""
    import torch
    from edge_to_b200 import _lib
    rng = np.random.default_rng(n)
    rho = rng.uniform(0.0, 1.0, n)
    dr = -np.exp(rng.normal(0.0, 3.0, n)) * (rng.uniform(size=n) < 0.9)
    dr[rng.uniform(size=n) < 0.01] = 1.0  # a positive sensitivity counts as zero
    A = 0.75
    ref, lam, steps = topopt.oc_update(rho, dr, A, A * n, vf, 0.2)
    r, d = torch.as_tensor(rho, device="cuda"), torch.as_tensor(dr, device="cuda")
    out = torch.empty_like(r)
    lo, so, ch = ctypes.c_double(), ctypes.c_int(), ctypes.c_double()
    _lib.call("edge_oc_update_static", n, _lib.ptr(r), _lib.ptr(d), A, A * n, vf, 0.2, _lib.ptr(out),
              ctypes.byref(lo), ctypes.byref(so), ctypes.byref(ch), _lib.stream_ptr())
    assert (lo.value, so.value) == (lam, steps)
    np.testing.assert_allclose(out.cpu().numpy(), ref, rtol=4e-16, atol=0)
    assert ch.value == pytest.approx(float(((ref - rho) ** 2).sum()), rel=1e-12)


@pytest.mark.parametrize("nel", [(1, 1), (31, 33), (32, 32), (70, 65), (1, 1, 1), (3, 2, 5), (4, 16, 32), (5, 17, 33),
                                 (9, 40, 31)])
@pytest.mark.parametrize("rmin", [1.0, 1.5, 2.0, 2.9, 5.5])
def test_filter_and_transpose_against_taps(nel, rmin):
    """H and H^T against the tap sums in numpy, where tiles end and at every halo width (5.5: the
    one-thread-per-element kernel, 2-D only).  At most 128 terms of order 1 per sum, whose weights add
    to 1: a few FP64 roundings."""
    import torch
    import edge_to_b200 as eb
    dim = len(nel)
    if rmin > 3.0 and dim == 3:
        pytest.skip("more taps than the filter takes")
    mesh = (eb.CuStructuredMesh2D if dim == 2 else eb.CuStructuredMesh3D)(*nel, *map(float, nel))
    flt = (eb.CuStructuredFilter2D if dim == 2 else eb.CuStructuredFilter3D)(mesh, rmin)
    rng = np.random.default_rng(7)
    x, y = rng.uniform(size=nel), rng.standard_normal(nel)
    offs, w = flt.offsets.cpu().numpy(), flt.weights.cpu().numpy()
    idx = np.stack(np.meshgrid(*[np.arange(n) for n in nel], indexing="ij"), -1).reshape(-1, dim)
    H = np.zeros((idx.shape[0], idx.shape[0]))
    for o, wk in zip(offs, w):
        nb = idx + o
        ok = np.all((nb >= 0) & (nb < np.array(nel)), axis=1)
        H[np.nonzero(ok)[0], np.ravel_multi_index(nb[ok].T, nel)] += wk
    H /= H.sum(axis=1, keepdims=True)
    fx = flt.dot(torch.as_tensor(x.ravel(), device="cuda")).cpu().numpy()
    ty = flt.T.dot(torch.as_tensor(y.ravel(), device="cuda")).cpu().numpy()
    np.testing.assert_allclose(fx, H @ x.ravel(), rtol=0, atol=2e-15)
    np.testing.assert_allclose(ty, H.T @ y.ravel(), rtol=0, atol=2e-14)


def _problem(nel, seed, h=None):
    import torch
    import edge_to_b200 as eb
    dim = len(nel)
    h = h or [1.0] * dim
    cls = eb.CuStructuredMesh2D if dim == 2 else eb.CuStructuredMesh3D
    mesh = cls(*nel, *[n * a for n, a in zip(nel, h)], stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))
    k = eb.CuStructuredStiffnessKernel(mesh)
    rng = np.random.default_rng(seed)
    n_dof = int(np.prod([v + 1 for v in nel])) * dim
    cons = rng.choice(n_dof, size=max(1, n_dof // 9), replace=False)
    E = rng.uniform(1e-9, 1.0, int(np.prod(nel)))
    u = rng.standard_normal(n_dof)
    k.set_rho(torch.as_tensor(E, device="cuda"))
    return mesh, k, cons, E, u


def _dense(mesh, nel, E, u, cons):
    """K(E) u and -u_e^T K0 u_e from the element matrix and the mesh's connectivity."""
    dim = len(nel)
    d = (np.asarray(mesh.elements)[:, :, None] * dim + np.arange(dim)).reshape(len(E), -1)
    K0 = np.asarray(mesh.K_single)
    v = u.copy()
    v[cons] = 0.0
    out = np.zeros_like(u)
    np.add.at(out, d.ravel(), (E[:, None] * (v[d] @ K0)).ravel())
    out[cons] = u[cons]
    return out, -np.einsum("ei,ij,ej->e", u[d], K0, u[d])


@pytest.mark.parametrize("nel", [(1, 1), (3, 4), (31, 3), (32, 33), (65, 130), (1, 1, 1), (2, 1, 3), (14, 5, 14), (15, 3, 15),
                                 (16, 7, 31), (37, 40, 17)])
@pytest.mark.parametrize("box", [False, True])
def test_product_and_energy_on_user_vectors(nel, box):
    """One-launch product and element energies where tiles end, on unit elements (the cube block form in
    3-D) and on boxes, with and without constraints, on a vector that is only 8-byte aligned, and with
    the product's own result as its input.  Entries of order 1 from at most 8 x 24 products of order
    1: FP64 roundings of the sum, 1e-14."""
    import torch
    mesh, k, cons, E, u = _problem(nel, 11, [1.0, 1.5, 0.75][:len(nel)] if box else None)
    ut = torch.as_tensor(u, device="cuda")
    odd = torch.empty(u.size + 1, dtype=torch.float64, device="cuda")[1:]
    odd.copy_(ut)
    for c in (np.zeros(0, dtype=np.int64), cons):
        k.set_constraints(c)
        ref, dk = _dense(mesh, nel, E, u, c)
        for x in (ut, odd):
            np.testing.assert_allclose(k.dot(x).cpu().numpy(), ref, rtol=0, atol=3e-14)
            np.testing.assert_allclose(k.process_grad(x).cpu().numpy(), dk, rtol=0, atol=1e-13)
        twice, _ = _dense(mesh, nel, E, ref, c)
        np.testing.assert_allclose(k.dot(k.dot(ut)).cpu().numpy(), twice, rtol=0, atol=2e-13)


@pytest.mark.parametrize("nel", [(2, 2), (6, 4), (12, 12), (14, 14), (16, 14), (30, 62), (62, 62), (4, 4, 4), (8, 6, 6),
                                 (10, 8, 8)])
def test_coarsest_inverse_solves_a_two_level_system(nel):
    """Coarsest matrices of 8 to 2,048 DOFs (blocks of 64: fewer, exactly one, two, one DOF more, many): the
    two-level V-cycle's PCG takes the oracle's iterations and reaches its solution, as it only does
    with the exact coarsest solve (rtol 1e-10; condition numbers below 1e5)."""
    import torch
    import edge_to_b200 as eb
    dim = len(nel)
    p = (topopt.mbb_problem if dim == 2 else topopt.cantilever_problem)(
        *nel, vf=0.4, mg_kwargs=dict(tol=1e-10, n_level=1, maxiter=300, variant="gpu"))
    E = np.random.default_rng(4).uniform(0.3, 1.0, p.grid.n_el) ** 3
    ref, _ = p.solver.solve(ops.assemble(p.grid, p.K0, E, p.cons), p.f, use_last=False)
    mesh = (eb.CuStructuredMesh2D if dim == 2 else eb.CuStructuredMesh3D)(
        *nel, *map(float, nel), stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))
    k = eb.CuStructuredStiffnessKernel(mesh)
    k.add_constraints(p.cons)
    sv = eb.CuMultiGrid(mesh, k, tol=1e-10, n_level=1, maxiter=300)
    x, res = sv.solve(torch.as_tensor(p.f, device="cuda"), torch.as_tensor(E, device="cuda"), use_last=False)
    assert res < 1e-10 and sv.last_iters == p.solver.pcg_iters[-1]
    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=0, atol=1e-9 * np.abs(ref).max())


@pytest.mark.parametrize("team", [1, 8])
@pytest.mark.parametrize("box", [True, False])
def test_batched_fine_operator_equals_the_per_problem_one(team, box, monkeypatch):
    """Grids that end at, before and after the marching operator's 30-node columns, of few and many rows,
    and an element matrix without the box structure (node-wise form): the batched FP64 solve takes the
    per-problem solver's iterations and reaches its compliances.  Both stop at a relative residual of
    1e-10, and a compliance's error is of the residual's second order: 1e-9 leaves the sums' roundings."""
    import edge_to_b200 as eb
    from edge_to_b200 import batch
    if not box:
        plain = eb.auto_stiffness

        def anisotropic(x, E, nu):
            K, D, B, A = plain(x, E, nu)
            v = np.asarray(K) @ np.arange(1.0, 9.0) ** 2 / 40.0  # in K's range: rigid motions stay free
            return K + 0.02 * np.outer(v, v), D, B, A
        monkeypatch.setattr(eb, "auto_stiffness", anisotropic)
    specs = [batch.random_spec(i, seed=9, nelx_range=(nx, nx), nely_range=(ny, ny))
             for i, (nx, ny) in enumerate([(28, 4), (30, 16), (32, 40), (58, 6), (60, 62), (62, 9), (120, 90)])]
    a = batch.BatchSIMP(specs, precision="fp64", tol=1e-10, maxiter=2000, n_threads=1)
    c = batch.BatchSIMP(specs, precision="fp64", tol=1e-10, maxiter=2000, persistent=True, team=team)
    a.step(2)
    c.step(2)
    for sp, ia, ic in zip(specs, a.items, c.items):
        assert ia["pcg"] == ic["pcg"], sp["index"]
        np.testing.assert_allclose(ic["comp"], ia["comp"], rtol=1e-9, atol=0)


@pytest.mark.parametrize("nel,n_level", [((2, 2), 1), ((8, 4), 2), ((64, 30), 1), ((62, 64), 1), ((126, 126), 1),
                                         ((128, 128), 2), ((48, 64), 4), ((128, 64), 6)])
@pytest.mark.parametrize("n_smooth", [1, 3])
def test_two_dimensional_cycle_below_the_fine_level(nel, n_level, n_smooth):
    """Level 1 of four nodes up to the last size that runs as one launch (4,096 nodes) and the first that
    does not, with levels of the whole cluster and of one block: the PCG takes the oracle's iterations
    to rtol 1e-10 and reaches its solution, as it only does with the oracle's cycle."""
    import torch
    import edge_to_b200 as eb
    p = topopt.mbb_problem(*nel, vf=0.4, mg_kwargs=dict(tol=1e-10, n_level=n_level, n_smooth=n_smooth, maxiter=600,
                                                        variant="gpu"))
    E = np.random.default_rng(4).uniform(0.3, 1.0, p.grid.n_el) ** 3
    ref, _ = p.solver.solve(ops.assemble(p.grid, p.K0, E, p.cons), p.f, use_last=False)
    mesh = eb.CuStructuredMesh2D(*nel, *map(float, nel), stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))
    k = eb.CuStructuredStiffnessKernel(mesh)
    k.add_constraints(p.cons)
    sv = eb.CuMultiGrid(mesh, k, tol=1e-10, n_level=n_level, n_smooth=n_smooth, maxiter=600)
    x, res = sv.solve(torch.as_tensor(p.f, device="cuda"), torch.as_tensor(E, device="cuda"), use_last=False)
    assert res < 1e-10 and sv.last_iters == p.solver.pcg_iters[-1]
    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=0, atol=1e-9 * np.abs(ref).max())


def _launches_per_iteration(nel, n_level, n_smooth, precision):
    import torch
    import edge_to_b200 as eb
    from edge_to_b200 import _lib
    mesh = eb.CuStructuredMesh2D(*nel, *map(float, nel), stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))
    k = eb.CuStructuredStiffnessKernel(mesh)
    left = np.arange(nel[1] + 1) * (nel[0] + 1)
    k.add_constraints(np.concatenate([2 * left, 2 * left + 1]))
    f = np.zeros(k.shape[0])
    f[-1] = -1.0
    f, E = torch.as_tensor(f, device="cuda"), torch.full((int(np.prod(nel)),), 0.5, dtype=torch.float64, device="cuda")
    last = None
    for its in range(2, 12):
        sv = eb.CuMultiGrid(mesh, k, tol=1e-300, n_level=n_level, n_smooth=n_smooth, maxiter=its, precision=precision,
                            tune_sweeps=False)
        counts = []
        for _ in range(3):  # the first solve may tune
            n = ctypes.c_longlong()
            sv.solve(f, E, use_last=False)
            _lib.call("edge_launch_count", k.handle, ctypes.byref(n))
            counts.append(n.value)
        assert sv.last_iters == its
        now = counts[2] - counts[1], sv.stats()["true_residuals"]
        if last and last[1] == now[1]:  # no residual replacement (mixed precision) in the added iteration
            return now[0] - last[0]
        last = now
    raise AssertionError("every iteration replaced the residual")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_coarsest_levels_stay_out_of_the_one_launch_cycle(precision):
    """The one-launch cycle runs on eight SMs, the dense product of a large coarsest level needs all of
    them (8,192 coarsest DOFs took 7.2 ms per iteration in one launch, 0.19 with separate ones).  A level
    between the transfers costs 2 n_smooth + 3 launches of its own where the cycle is separate, none where
    it is one launch."""
    for ns in (1, 3):
        one = _launches_per_iteration((96, 96), 1, ns, precision)    # 4,802 coarsest DOFs
        two = _launches_per_iteration((96, 96), 2, ns, precision)    # 1,250
        assert two - one == 2 * ns + 3
    three = _launches_per_iteration((64, 64), 3, 3, precision)       # 162 coarsest DOFs: one launch
    assert three < two


@pytest.mark.parametrize("threads", [512, 1024])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batched_result_does_not_depend_on_the_company(precision, threads):
    """Three SIMP iterations of the same problems, alone and in two companies, by teams of 1 to 16 blocks
    (chosen per problem with team > 1; split_dof = 1 keeps the caller's team): the same bits, as every
    step of a solve is node by node and its sums have one order.  Sizes from less than one to several
    of a block's passes over the nodes."""
    import torch
    from edge_to_b200 import batch
    specs = [batch.random_spec(i, seed=21, nelx_range=(nx, nx), nely_range=(ny, ny))
             for i, (nx, ny) in enumerate([(24, 8), (60, 20), (64, 40), (120, 44), (200, 90), (300, 120)])]

    def run(which, **kw):
        b = batch.BatchSIMP([specs[i] for i in which], precision=precision, tol=1e-6, maxiter=400, persistent=True,
                            block_threads=threads, **kw)
        b.step(3)
        return {i: (it["rho"].cpu(), it["dr"].cpu(), u.cpu(), it["comp"], it["pcg"])
                for i, it, u in zip(which, b.items, b.batch.U)}
    ref = run(range(6), team=1)
    others = [run(range(6), team=4), run([5, 0, 2], team=8), run([1, 3, 4], team=2, split_dof=1)]
    others += [run([i], team=4) for i in (0, 3, 5)]
    for o in others:
        for i, got in o.items():
            for a, b in zip(got[:3], ref[i][:3]):
                assert torch.equal(a, b), i
            assert got[3:] == ref[i][3:], i


@pytest.mark.parametrize("nelx", [458744, 458745, 524280, 524281])
def test_product_and_energy_of_very_long_bars(nelx):
    """One row of elements around the lengths at which the one-launch product (tiles of 7 node columns) and
    energies (8 element columns) reach the limit of 65,535 tiles: beyond it the calls take the converting
    path.  FP64 roundings of sums of at most 8 x 24 products of order 1."""
    import torch
    nel = (nelx, 1, 1)
    mesh, k, cons, E, u = _problem(nel, 5)
    k.set_constraints(cons)
    ref, dk = _dense(mesh, nel, E, u, cons)
    ut = torch.as_tensor(u, device="cuda")
    np.testing.assert_allclose(k.dot(ut).cpu().numpy(), ref, rtol=0, atol=3e-14)
    np.testing.assert_allclose(k.process_grad(ut).cpu().numpy(), dk, rtol=0, atol=1e-13)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_default_kernel_of_a_medium_stencil_level(precision):
    """Level 1 of 34,848 slots: one thread per node in FP64 (10.6 us a sweep against 12.3), a warp per
    direction in mixed precision (8.5 against 10.3).  The two add a node's terms in different orders, so
    the bits of a solve tell which one the default took."""
    import torch
    import edge_to_b200 as eb
    from edge_to_b200 import _lib
    nel = (64, 64, 56)
    mesh, k, _, E, _ = _problem(nel, 2)
    k.set_constraints(np.arange(3 * 65 * 57))
    f = np.zeros(k.shape[0])
    f[-1] = -1.0
    f = torch.as_tensor(f, device="cuda")
    got = []
    for quad in (None, 20000, 60000):
        sv = eb.CuMultiGrid(mesh, k, tol=1e-300, n_level=3, maxiter=3, precision=precision, autotune=False,
                            tune_sweeps=False)
        if quad is not None:
            _lib.call("edge_set_stencil_quad", k.handle, quad)
        got.append(sv.solve(f, torch.as_tensor(E, device="cuda"), use_last=False)[0].cpu())
    assert not torch.equal(got[1], got[2])
    assert torch.equal(got[0], got[1 if precision == "fp64" else 2])


@pytest.mark.parametrize("nel,n_level", [((16, 14), 1), ((62, 62), 1), ((64, 32), 2), ((10, 8, 8), 1), ((16, 8, 8), 2)])
def test_coarsest_inverse_with_void_elements(nel, n_level):
    """A block of void elements (1e-9) in a solid grid: the pivots of the block sweeps span the contrast.
    The PCG takes the oracle's iterations; the solutions then differ by roundings of the contrast at most
    (1e9 machine roundings of the largest displacement, 1e-6)."""
    import torch
    import edge_to_b200 as eb
    dim = len(nel)
    p = (topopt.mbb_problem if dim == 2 else topopt.cantilever_problem)(
        *nel, vf=0.4, mg_kwargs=dict(tol=1e-8, n_level=n_level, maxiter=1000, variant="gpu"))
    E = np.ones(nel)
    E[tuple(slice(n // 4, n // 2) for n in nel)] = 1e-9
    E = E.ravel()
    ref, _ = p.solver.solve(ops.assemble(p.grid, p.K0, E, p.cons), p.f, use_last=False)
    mesh = (eb.CuStructuredMesh2D if dim == 2 else eb.CuStructuredMesh3D)(
        *nel, *map(float, nel), stiffness=lambda x: eb.auto_stiffness(x, 1.0, 0.3))
    k = eb.CuStructuredStiffnessKernel(mesh)
    k.add_constraints(p.cons)
    sv = eb.CuMultiGrid(mesh, k, tol=1e-8, n_level=n_level, maxiter=1000)
    x, res = sv.solve(torch.as_tensor(p.f, device="cuda"), torch.as_tensor(E, device="cuda"), use_last=False)
    assert res < 1e-8 and sv.last_iters == p.solver.pcg_iters[-1]
    np.testing.assert_allclose(x.cpu().numpy(), ref, rtol=0, atol=1e-6 * np.abs(ref).max())


@pytest.mark.parametrize("nel", [(40, 37), (9, 20, 33)])
@pytest.mark.parametrize("rmin", [1.0, 1.5, 2.0, 2.9])
def test_filter_keeps_an_infinity_to_its_taps(nel, rmin):
    """An infinite value reaches exactly the elements that have a tap on it: a tap that the stencil does
    not have is not a product with zero.  The others as in the finite test."""
    import torch
    import edge_to_b200 as eb
    dim = len(nel)
    mesh = (eb.CuStructuredMesh2D if dim == 2 else eb.CuStructuredMesh3D)(*nel, *map(float, nel))
    flt = (eb.CuStructuredFilter2D if dim == 2 else eb.CuStructuredFilter3D)(mesh, rmin)
    x = np.random.default_rng(3).uniform(size=nel)
    x[tuple(n // 2 for n in nel)] = np.inf
    x[tuple(0 for _ in nel)] = np.inf
    offs, w = flt.offsets.cpu().numpy(), flt.weights.cpu().numpy()
    idx = np.stack(np.meshgrid(*[np.arange(n) for n in nel], indexing="ij"), -1)
    num, norm = np.zeros(nel), np.zeros(nel)
    for o, wk in zip(offs, w):
        nb = idx + o
        ok = np.all((nb >= 0) & (nb < np.array(nel)), axis=-1)
        num[ok] += wk * x[tuple(nb[ok].T)]
        norm[ok] += wk
    trans = np.zeros(nel)
    for o, wk in zip(offs, w):
        nb = idx + o
        ok = np.all((nb >= 0) & (nb < np.array(nel)), axis=-1)
        trans[ok] += wk / norm[tuple(nb[ok].T)] * x[tuple(nb[ok].T)]
    xt = torch.as_tensor(x.ravel(), device="cuda")
    for got, ref, atol in ((flt.dot(xt), num / norm, 2e-15), (flt.T.dot(xt), trans, 2e-14)):
        got, ref = got.cpu().numpy(), ref.ravel()
        np.testing.assert_array_equal(np.isinf(got), np.isinf(ref))
        assert not np.isnan(got).any()
        f = np.isfinite(ref)
        np.testing.assert_allclose(got[f], ref[f], rtol=0, atol=atol)
