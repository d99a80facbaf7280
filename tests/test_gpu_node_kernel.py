"""The node kernel (every bath coupling at any N) at the edges of its tiles:
one and several rounds of elements per thread, one node per tile, more baths
than are staged at once, partial last tiles, against the CPU oracle.

FP64: 1e-12 of the output scale for one apply, 1e-10 for a propagated state."""
import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

PROBLEMS = [
    ("indep_n9_K2", dict(kind="independent", n=9, matsubara=2, truncation=4)),
    ("indep_n13_K1_complex", dict(kind="independent", n=13, matsubara=1, truncation=3, complex_h=True)),
    ("indep_n33_K1", dict(kind="independent", n=33, matsubara=1, truncation=3)),
    ("indep_n48_K1", dict(kind="independent", n=48, matsubara=1, truncation=2)),
    ("indep_n3_K5", dict(kind="independent", n=3, matsubara=5, truncation=4)),
    ("indep_n4_K4_unnormalized", dict(kind="independent", n=4, matsubara=4, truncation=3, normalized=False)),
    ("diag_n2_b1_L40", dict(kind="diagonal", n=2, matsubara=1, truncation=41, baths=1)),
    ("diag_n9_b4_K2_complex", dict(kind="diagonal", n=9, matsubara=2, truncation=4, baths=4, complex_h=True)),
    ("diag_n24_b1_K1", dict(kind="diagonal", n=24, matsubara=1, truncation=5, baths=1)),
    ("diag_n4_b9_K3", dict(kind="diagonal", n=4, matsubara=3, truncation=3, baths=9)),
    ("full_n2_b9_K1", dict(kind="full", n=2, matsubara=1, truncation=4, baths=9)),
    ("full_n6_b3_K2", dict(kind="full", n=6, matsubara=2, truncation=5, baths=3)),
    ("full_n11_b2_K5_complex", dict(kind="full", n=11, matsubara=5, truncation=3, baths=2, complex_h=True)),
    ("full_n32_b3_K1", dict(kind="full", n=32, matsubara=1, truncation=3, baths=3)),
    ("full_n5_vacuum", dict(kind="full", n=5, matsubara=1, truncation=1, baths=2)),
]


@pytest.mark.parametrize("name,kw", PROBLEMS, ids=[p[0] for p in PROBLEMS])
def test_apply_matches_oracle(name, kw):
    p = cases.random_problem(seed=7, **kw)
    o = O.Oracle(p)
    s = cases.random_hermitian_state(o.M, p.num_states, seed=2)
    ref = o.apply(s)
    with Hierarchy(p) as h:
        got = h.apply(s)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    d = got.view(np.complex128).reshape(-1, p.num_states, p.num_states)
    assert np.array_equal(d, np.conj(np.transpose(d, (0, 2, 1))))


@pytest.mark.parametrize("name", ["indep_n9_K2", "diag_n9_b4_K2_complex", "full_n6_b3_K2", "full_n32_b3_K1"])
def test_integrators_match_oracle(name):
    p = cases.random_problem(seed=7, **dict(PROBLEMS)[name])
    p.fix_incompatible_combinations("rkf45")
    o = O.Oracle(p)
    ref, steps, _, _ = o.rk4(o.initial_state(), 0.0002, 0.004)
    with Hierarchy(p) as h:
        assert h.rk4(0.0002, 0.004)[0] == steps
        assert np.abs(h.get_state() - ref).max() <= 1e-10
        h.reset()
        ref, st, *_ = o.rkf45(o.initial_state(), 0.0002, 0.004, 1e-6, 1e-6)
        assert h.rkf45(0.0002, 0.004, 1e-6, 1e-6)["steps"] == st["steps"]
        assert np.abs(h.get_state() - ref).max() <= 1e-10
