"""A batch's schedule can be set back to the untuned one (as many CTAs per SM
as fit); what lies outside the range is refused."""
import numpy as np
import pytest

from phi_b200 import capi, configs
from phi_b200.heom import Batch

pytestmark = pytest.mark.gpu


def test_back_to_the_untuned_schedule():
    probs = configs.batched(seed=17, count=8, budget_bytes=2**20, depth_range=(2, 5))
    with Batch(probs) as b:
        b.rk4(0.0005, 20)
        b.set_schedule(1, 0)
        b.rk4(0.0005, 20)
        b.set_schedule(0, 1)
        b.rk4(0.0005, 20)
        got = [b[i].get_state() for i in range(b.count)]
        for cps, order in ((-1, 0), (33, 0), (0, 2), (0, -1)):
            with pytest.raises(capi.PhiError) as e:
                b.set_schedule(cps, order)
            assert e.value.code == capi.PHI_E_INVALID
    with Batch(probs) as b:
        b.rk4(0.0005, 60)
        for i in range(b.count):
            assert np.array_equal(got[i], b[i].get_state())
