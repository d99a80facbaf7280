"""The time-local term by element, exchanged between the transposed elements
(tile kernel from 4 sites on, RKF45 from 10; node kernel from 9), and by pairs
below: every shape over a hierarchy with a partial last tile, where most nodes
are in the deepest tier, RK4 and RKF45 against the CPU oracle (state within 1e-10
of its largest element), mixed precision against FP64 (rho_0 within 1e-6)."""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200 import capi
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

SIZES = [(2, 3), (3, 1), (4, 1), (4, 3), (5, 2), (6, 1), (7, 2), (8, 3), (9, 1), (9, 2), (10, 1), (10, 3), (11, 1),
         (12, 2), (16, 1), (16, 2), (20, 1), (24, 1), (33, 1), (3, 4)]


@pytest.mark.parametrize("filtered", [False, True], ids=["plain", "filtered"])
@pytest.mark.parametrize("n,k1", SIZES)
def test_time_local_runs(n, k1, filtered):
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=3 if n < 16 else 2, seed=3 * n + k1,
                             scale=20.0, complex_h=n in (5, 11))
    p.use_time_local_truncation = True
    p.filter_tolerance = 1e-7 if filtered else 0.0
    p.fix_incompatible_combinations("rkf45")
    dt, t_end = 1e-4, 3.5e-4
    with Hierarchy(p) as h:
        o = O.Oracle(p)
        ref, steps, _, _ = o.rk4(o.initial_state(), dt, t_end)
        assert h.rk4(dt, t_end)[0] == steps
        assert np.abs(h.get_state() - ref).max() <= 1e-10 * np.abs(ref).max()
        rho = h.rho0()
    with Hierarchy(p) as h:
        o = O.Oracle(p)
        ref, st = o.rkf45(o.initial_state(), dt, t_end, 1e-6, 1e-7)[:2]
        assert h.rkf45(dt, t_end, 1e-6, 1e-7)["steps"] == st["steps"]
        assert np.abs(h.get_state() - ref).max() <= 1e-10 * np.abs(ref).max()
    if n in (2, 3, 4, 5, 6, 7, 8, 10, 12, 16, 24) and k1 <= 3:
        with Hierarchy(p, precision=capi.PHI_PREC_MIXED) as h:
            h.rk4(dt, t_end)
            assert np.abs(h.rho0() - rho).max() <= 1e-6


@pytest.mark.parametrize("n", [3, 4, 9, 16])
def test_single_tier(n):
    """One tier: every node is deepest and there are no neighbour terms."""
    p = cases.random_problem("independent", n=n, matsubara=1, truncation=1, seed=n, scale=20.0)
    p.use_time_local_truncation = True
    p.fix_incompatible_combinations("rkf45")
    with Hierarchy(p) as h:
        o = O.Oracle(p)
        ref, *_ = o.rk4(o.initial_state(), 1e-4, 9.5e-4)
        h.rk4(1e-4, 9.5e-4)
        assert np.abs(h.get_state() - ref).max() <= 1e-10 * np.abs(ref).max()
