"""RKF45 of 10 sites and more over three and four tiers, where the neighbour terms
are summed by element (and by the node kernel) in another order than below 10
sites: the oracle's accepted and rejected steps, the run ends at t_end, the state
within 1e-10; in mixed precision the run ends at t_end with rho_0 within 1e-6."""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200 import capi
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

T_END = 0.02


@pytest.mark.parametrize("n,k1,depth", [(10, 2, 3), (10, 1, 4), (12, 2, 3), (16, 1, 3), (24, 1, 2), (9, 2, 3), (13, 1, 3)])
def test_ends_like_the_oracle(n, k1, depth):
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=depth + 1, seed=n, scale=100.0)
    p.fix_incompatible_combinations("rkf45")
    o = O.Oracle(p)
    ref, st, *_ = o.rkf45(o.initial_state(), 0.001, T_END, 1e-6, 1e-6)
    assert abs(st["final_time"] - T_END) <= 1e-15
    with Hierarchy(p) as h:
        got = h.rkf45(0.001, T_END, 1e-6, 1e-6)
        assert (got["steps"], got["accepted"]) == (st["steps"], st["accepted"])
        assert got["final_time"] == st["final_time"]
        assert np.abs(h.get_state() - ref).max() <= 1e-10
    if n in (9, 13):
        return
    with Hierarchy(p, precision=capi.PHI_PREC_MIXED) as h:
        assert abs(h.rkf45(0.001, T_END, 1e-6, 1e-6)["final_time"] - T_END) <= 1e-15
        assert np.abs(h.rho0() - o.rho0(ref)).max() <= 1e-6
