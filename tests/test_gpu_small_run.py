"""The one-CTA RK4 run (heom_small.cu) at the edges of its register rows:
every compiled row size, real and complex Hamiltonians, one item more than
threads, rows kept and continued runs, against the CPU oracle (1e-10; PHI's
unnormalised diagonal hierarchies relative to their largest element)."""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

# kind, n, baths, K+1, depth
SIZES = [("diagonal", 2, 1, 1, 10), ("diagonal", 2, 1, 1, 84), ("diagonal", 2, 1, 1, 85), ("diagonal", 2, 2, 1, 4),
         ("diagonal", 2, 1, 3, 3), ("diagonal", 3, 1, 2, 4), ("diagonal", 3, 2, 1, 5), ("diagonal", 4, 2, 2, 2),
         ("diagonal", 5, 3, 2, 1), ("independent", 2, 2, 4, 1), ("independent", 3, 3, 4, 1)]


@pytest.mark.parametrize("complex_h", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("kind,n,baths,k1,depth", SIZES)
def test_run_matches_oracle(kind, n, baths, k1, depth, complex_h):
    p = cases.random_problem(kind, n=n, baths=baths, matsubara=k1, truncation=depth + 1, seed=depth + n,
                             complex_h=complex_h)
    dt = 0.0002
    o = O.Oracle(p)
    ref, steps, times, rows = o.rk4(o.initial_state(), dt, 30.5 * dt, output_min_step=4 * dt, capacity=40)
    with Hierarchy(p) as h:
        n1, t1, r1 = h.rk4(dt, 30.5 * dt, output_min_step=4 * dt, capacity=40)
        assert n1 == steps and np.array_equal(t1, times)
        assert np.abs(r1 - rows).max() <= 1e-10
        assert np.abs(h.get_state() - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
