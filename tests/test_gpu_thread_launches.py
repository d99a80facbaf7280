"""Launches of one kernel from several threads, each thread with problems of
another size: a thread's smaller problem leaves the kernel's shared-memory
limit where the larger problem of another thread needs it; and a thread's first
launch inside a stream capture."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import torch

import cases
from phi_b200.heom import Hierarchy

pytestmark = pytest.mark.gpu


def _node(n):  # more than 48 KiB per CTA from N = 24 on
    p = cases.random_problem("full", n=n, matsubara=1, truncation=3, baths=3, seed=n)

    def run():
        with Hierarchy(p) as h:
            return h.apply(cases.random_hermitian_state(h.num_nodes, n, seed=1))
    return run


def _tile(depth):  # the prefactor tables grow with the depth
    p = cases.random_problem("independent", n=16, matsubara=1, truncation=depth + 1, seed=2)
    p.fix_incompatible_combinations("rkf45")

    def run():
        with Hierarchy(p) as h:
            h.rkf45(1e-4, 2e-3, 1e-6, 1e-6)
            return h.get_state()
    return run


@pytest.mark.parametrize("large,small", [(_node(32), _node(24)), (_tile(3), _tile(1))], ids=["node", "tile"])
def test_a_smaller_problem_on_another_thread(large, small):
    with ThreadPoolExecutor(1) as a, ThreadPoolExecutor(1) as b:
        ref = a.submit(large).result()
        assert np.isfinite(b.submit(small).result()).all()
        got = a.submit(large).result()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("kind,n", [("full", 26), ("independent", 13), ("diagonal", 3), ("independent", 12)])
def test_first_apply_of_a_thread_under_capture(kind, n):
    """The limit is raised by a thread's first launch, which may be captured."""
    p = cases.random_problem(kind, n=n, matsubara=2, truncation=3, seed=5, **({} if kind == "independent" else {"baths": 3}))
    with Hierarchy(p) as h:
        s = cases.random_hermitian_state(h.num_nodes, n, seed=4)
        x = torch.from_numpy(s).cuda()
        y = torch.zeros_like(x)

        def captured():
            torch.cuda.set_device(0)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                h._check(h.lib.phi_gpu_apply_device(h.ctx, x.data_ptr(), y.data_ptr(),
                                                    torch.cuda.current_stream().cuda_stream))
            graph.replay()
            torch.cuda.synchronize()
        with ThreadPoolExecutor(1) as a:
            a.submit(captured).result()
        assert np.array_equal(y.cpu().numpy(), h.apply(s))
