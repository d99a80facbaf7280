"""RK4 stages that overlap (each kernel's start with the last tiles of the one
before) at the edges of one tile per CTA, and the batch's untuned schedule (as
many CTAs per SM as fit): the same state bit for bit whatever the grid."""
import numpy as np
import pytest

import cases
from phi_b200 import capi, configs
from phi_b200.heom import Batch, Hierarchy

pytestmark = pytest.mark.gpu

PRECISIONS = pytest.mark.parametrize("precision", [capi.PHI_PREC_FP64, capi.PHI_PREC_MIXED], ids=["fp64", "mixed"])


# At one CTA per SM: fewer tiles than SMs, just more (some CTAs have a second
# tile), several per CTA.  21 steps: a graph replay and direct launches.
@PRECISIONS
@pytest.mark.parametrize("n,k1,depth", [(3, 2, 8), (3, 2, 9), (4, 2, 7), (16, 1, 3), (2, 3, 10)])
def test_rk4_bits_do_not_depend_on_the_grid(n, k1, depth, precision):
    p = cases.random_problem("independent", n=n, matsubara=k1, truncation=depth + 1, seed=n + depth)
    out = []
    for cps in (0, 1):
        with Hierarchy(p, precision=precision) as h:
            h.set_tile_schedule(h.tile_schedule()["threads"], cps)
            h.rk4(1e-4, 20.5e-4)
            out.append(h.get_state())
    assert np.isfinite(out[0].view(np.float64)).all()
    assert np.array_equal(out[0], out[1])


@PRECISIONS
@pytest.mark.parametrize("count", [1, 16])
def test_untuned_batch_equals_a_set_schedule(count, precision):
    probs = configs.batched(seed=17, count=count, budget_bytes=2**20, depth_range=(2, 6))
    with Batch(probs, precision=precision) as b:
        b.rk4(0.0005, 20)
        b.set_schedule(1, 1)  # drops the graph captured for the untuned grid
        b.rk4(0.0005, 20)
        got = [b[i].get_state() for i in range(b.count)]
    with Batch(probs, precision=precision) as b:
        b.set_schedule(1, 1)
        b.rk4(0.0005, 40)
        ref = [b[i].get_state() for i in range(b.count)]
    for a, r in zip(got, ref):
        assert np.array_equal(a, r)
