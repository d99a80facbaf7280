"""Full couplings whose operators do not all fit shared memory at once (large N
with several baths, many baths at a moderate N): one apply, RK4, RKF45 and the
time-local truncation against the CPU oracle.

An element of an apply is a sum of n = nb (4 N + 4 (K + 1)) rounded products,
so its error is at most n 2^-53 times the sum of their magnitudes, which for
terms of random sign is about sqrt(n) times the output's scale.  A state
propagated over 5 steps of dt |L| < 1 adds 30 such applies of a state of order
one: 1e-10."""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

# (N, baths): the largest N of the coupling kind with one to eight baths, and
# bath counts past what each N holds at once.
SIZES = [(49, 1), (49, 8), (48, 5), (40, 11), (32, 21), (30, 32), (24, 42), (19, 64)]


def _problem(n, nb, **kw):
    return cases.random_problem("full", n=n, matsubara=1, truncation=2, baths=nb, seed=n + nb, **kw)


@pytest.mark.parametrize("complex_h", [False, True], ids=["real", "complex"])
@pytest.mark.parametrize("n,nb", SIZES)
def test_apply_matches_oracle(n, nb, complex_h):
    p = _problem(n, nb, complex_h=complex_h)
    o = O.Oracle(p)
    s = cases.random_hermitian_state(o.M, n, seed=3)
    ref = o.apply(s)
    with Hierarchy(p) as h:
        got = h.apply(s)
    terms = nb * (4 * n + 4)
    assert np.abs(got - ref).max() <= terms ** 1.5 * 2.0 ** -53 * np.abs(ref).max()


@pytest.mark.parametrize("time_local", [False, True], ids=["plain", "time_local"])
@pytest.mark.parametrize("n,nb", [(48, 5), (30, 32), (19, 64)])
def test_integrators_match_oracle(n, nb, time_local):
    p = _problem(n, nb, scale=10.0)
    p.use_time_local_truncation = time_local
    p.fix_incompatible_combinations("rkf45")
    dt = 2e-5
    with Hierarchy(p) as h:
        o = O.Oracle(p)
        ref, steps, _, _ = o.rk4(o.initial_state(), dt, 4.5 * dt)
        assert h.rk4(dt, 4.5 * dt)[0] == steps == 5
        assert np.abs(h.get_state() - ref).max() <= 1e-10
        h.reset()
        o = O.Oracle(p)
        ref, st, *_ = o.rkf45(o.initial_state(), dt, 4.5 * dt, 1e-6, 1e-7)
        assert h.rkf45(dt, 4.5 * dt, 1e-6, 1e-7)["steps"] == st["steps"]
        assert np.abs(h.get_state() - ref).max() <= 1e-10
