"""Element-wise passes on user-layout arrays (csrc/fields.cu) against the CPU oracle, at the
sizes where their tiles and blocks end."""
import ctypes

import numpy as np
import pytest

from oracle import topopt

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
