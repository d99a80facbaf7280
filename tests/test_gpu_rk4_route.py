"""Which way RK4 runs are taken: in one cluster where a hierarchy's tiles fit one,
by a launch per stage from the first size that does not, in one CTA for small
couplings off the tiled sizes; cluster runs against the CPU oracle (FP64: 1e-10
of a state of order one; mixed: rho_0 within 1e-6, the mode's target); and the
RKF45 stages' own schedule."""
import ctypes

import numpy as np
import pytest

import cases
from oracle import oracle as O
from phi_b200 import capi, configs
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu

NONE, STAGES, CTA, CLUSTER = range(4)
FP64, MIXED = capi.PHI_PREC_FP64, capi.PHI_PREC_MIXED


def _route(h):
    out = ctypes.c_int32(-1)
    capi.check(h.lib.phi_gpu_debug_get_rk4_route(h.ctx, ctypes.byref(out)))
    return out.value


def _cluster_nodes(n, mixed):
    """Nodes a cluster holds: 16 CTAs of 256 threads with at most 32 bytes of
    elements per thread and operand, at most 64 nodes each."""
    return 16 * min(64, (4 if mixed else 2) * (256 // n) // n)


SIZES = [(2, 1, 2), (2, 3, 5), (3, 2, 3), (3, 2, 5), (3, 2, 6), (4, 2, 4), (4, 2, 5), (5, 2, 3), (5, 2, 4), (6, 1, 4),
         (7, 2, 2), (8, 1, 3), (10, 1, 2), (12, 1, 2), (16, 1, 1), (16, 1, 2), (24, 1, 1)]


@pytest.mark.parametrize("precision", [FP64, MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("n,k1,depth", SIZES)
def test_tiled_sizes(n, k1, depth, precision):
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=depth + 1, seed=n + depth, scale=20.0)
    o = O.Oracle(p)
    ref, steps, _, _ = o.rk4(o.initial_state(), 0.0005, 0.00475)
    with Hierarchy(p, precision=precision) as h:
        assert _route(h) == NONE
        assert h.rk4(0.0005, 0.00475)[0] == steps
        fits = n < 24 and h.num_nodes <= _cluster_nodes(n, precision == MIXED)
        assert _route(h) == (CLUSTER if fits else STAGES)
        if precision == FP64:
            assert np.abs(h.get_state() - ref).max() <= 1e-10
        assert np.abs(h.rho0() - o.rho0(ref)).max() <= (1e-10 if precision == FP64 else 1e-6)


def test_other_routes():
    small = cases.random_problem("diagonal", n=2, matsubara=1, truncation=4, baths=1, seed=1)
    big = cases.random_problem("full", n=3, matsubara=2, truncation=4, baths=2, seed=1)
    for p, route in ((small, CTA), (big, STAGES)):
        with Hierarchy(p) as h:
            h.rk4(0.0005, 0.002)
            assert _route(h) == route
    # What changes between stages keeps a small tiled hierarchy on launches.
    for change in ("filter", "time_local", "annealing"):
        p = cases.random_problem("independent", n=3, matsubara=1, truncation=4, seed=1)
        if change == "filter":
            p.filter_tolerance = 1e-6
        elif change == "time_local":
            p.use_time_local_truncation = True
        else:
            p = cases.annealed(p, 0.01)
        with Hierarchy(p) as h:
            h.rk4(0.0005, 0.002)
            assert _route(h) == STAGES, change


def test_rkf45_schedule():
    def schedule(h):
        threads, cps = ctypes.c_int32(-1), ctypes.c_int32(-1)
        capi.check(h.lib.phi_gpu_debug_get_rkf45_schedule(h.ctx, ctypes.byref(threads), ctypes.byref(cps)))
        return threads.value, cps.value

    p = configs.frenkel7()  # tuned: more than 2^20 elements
    p.fix_incompatible_combinations("rkf45")
    with Hierarchy(p, precision=MIXED) as h:
        assert schedule(h) == (0, 0)
        st = h.rkf45(0.001, 0.005, 1e-6, 1e-6)
        ref, (threads, cps) = h.get_state(), schedule(h)
        assert threads in (256, 320) and cps >= 0
        for other in ((256, 0), (320, 0), (320, 1)):
            h.set_tile_schedule(*other)
            assert schedule(h) == other
            h.reset()
            assert h.rkf45(0.001, 0.005, 1e-6, 1e-6)["steps"] == st["steps"]
            assert np.array_equal(h.get_state(), ref)
    p = configs.frenkel7(depth=3)  # too small to be tuned
    p.fix_incompatible_combinations("rkf45")
    with Hierarchy(p) as h:
        h.rkf45(0.001, 0.005, 1e-6, 1e-6)
        assert schedule(h) == (0, 0)
