"""The tile kernel's element and pair mappings at the edges of their tiles:
every tiled N with K+1 = 1..3 over a hierarchy whose last tile is partial and
one smaller than a tile, in both arithmetics, against the CPU oracle.

FP64: 1e-12 of the output scale.  Mixed: an element is a sum of at most
2N + 4(K+1) + 1 rounded products, each within 2^-24 of its value (and of the
complex64 input's rounding), so 2e-6 of the output scale.
"""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200 import capi
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

SIZES = [(n, k1) for n in (2, 3, 4, 5, 6, 7, 8, 10, 12, 16, 24) for k1 in (1, 2, 3) if n * k1 <= 48]


@pytest.mark.parametrize("n,k1", SIZES)
@pytest.mark.parametrize("complex_h", [False, True], ids=["real", "complex"])
def test_apply_of_partial_tiles(n, k1, complex_h):
    for depth in (1, 3 if n * k1 <= 12 else 2):
        p = cases.random_problem("independent", n=n, matsubara=k1, truncation=depth + 1, seed=n + k1,
                                 complex_h=complex_h)
        o = O.Oracle(p)
        s = cases.random_hermitian_state(o.M, n, seed=depth)
        ref = o.apply(s)
        scale = np.abs(ref).max()
        for precision, tol in ((capi.PHI_PREC_FP64, 1e-12), (capi.PHI_PREC_MIXED, 2e-6)):
            with Hierarchy(p, precision=precision) as h:
                assert np.abs(h.apply(s) - ref).max() <= tol * scale, (depth, precision)


@pytest.mark.parametrize("n,k1", [(3, 3), (8, 2), (10, 2), (16, 1), (24, 1)])
def test_integrators_on_both_mappings(n, k1):
    """RKF45 (pairs below N = 10) and RK4 over two tiers: the oracle's steps,
    its state within 1e-10."""
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=3, seed=n)
    o = O.Oracle(p)
    ref, steps, _, _ = o.rk4(o.initial_state(), 0.0005, 0.01)
    with Hierarchy(p) as h:
        assert h.rk4(0.0005, 0.01)[0] == steps
        assert np.abs(h.get_state() - ref).max() <= 1e-10
        h.reset()
        ref, steps, *_ = o.rkf45(o.initial_state(), 0.0005, 0.02, 1e-6, 1e-6)
        assert h.rkf45(0.0005, 0.02, 1e-6, 1e-6)["steps"] == steps["steps"]
        assert np.abs(h.get_state() - ref).max() <= 1e-10
