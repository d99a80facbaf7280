"""The resident RK4 run (one cluster for the whole run of a small tiled
hierarchy) against the launch-per-stage path: the same state bit for bit, at
one tile, a partial last tile, every cluster size and the first hierarchy that
is too large for a cluster; rows and their times; a run continued by another."""
import numpy as np
import pytest

import cases
from phi_b200 import capi
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

SIZES = [(2, 1, 2), (2, 3, 5), (3, 1, 3), (3, 2, 3), (3, 2, 5), (4, 3, 3), (5, 2, 2), (6, 1, 4), (7, 2, 2), (8, 1, 3),
         (10, 1, 2), (12, 2, 1), (16, 1, 1), (4, 2, 5)]


def _run(p, precision, staged, steps):
    with Hierarchy(p, precision=precision) as h:
        if staged:  # a bounded-wait limit keeps the run on the launch-per-stage path
            capi.check(h.lib.phi_gpu_debug_set_wait_limit(h.ctx, 1 << 22))
        a = h.rk4(0.0005, (steps - 0.5) * 0.0005, output_min_step=0.001, capacity=steps)
        b = h.rk4(0.0005, h.time + 4.5 * 0.0005)  # continues
        return h.get_state(), a, b[0], h.time


@pytest.mark.parametrize("precision", [capi.PHI_PREC_FP64, capi.PHI_PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,k1,depth", SIZES)
def test_same_bits_as_launches(n, k1, depth, precision):
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=depth + 1, seed=n + depth,
                             complex_h=n == 5)
    s0, a0, n0, t0 = _run(p, precision, True, 21)
    s1, a1, n1, t1 = _run(p, precision, False, 21)
    assert np.array_equal(s0, s1)
    assert a0[0] == a1[0] and n0 == n1 and t0 == t1
    assert np.array_equal(a0[1], a1[1]) and np.array_equal(a0[2], a1[2])
