"""A steady-state solve that stops inside an outer iteration leaves the last
iterate in the context, the BiCG steps it has taken included.

The problem makes that exact: H = 0, one tier, every bath with the same
gamma = 8.  From rho_0 = I/N the residual lives in the elements (m, m) of the
first tier, eigenvectors of the operator with eigenvalue -8, so the first BiCG
step gives x exactly (products and quotients of powers of two do not round),
the residual becomes zero and the next inner product is a breakdown."""
import numpy as np
import pytest

from phi_b200 import capi
from phi_b200.heom import Hierarchy, PhiParameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ell", [1, 2, 3])
@pytest.mark.parametrize("n", [2, 9], ids=["tile", "node"])
def test_last_iterate_after_a_breakdown(n, ell):
    p = PhiParameters(num_states=n, time_indepenent_hamiltonian=np.zeros((n, n), np.complex128),
                      num_bath_couplings=n, num_matsubara_terms=1, hierarchy_truncation_level=2, temperature=300.0,
                      gamma=np.full(n, 8.0), lambda_=np.linspace(20.0, 40.0, n))
    rho = np.zeros((n, n), np.complex128)
    rho[0, 0] = 1.0
    p.initial_density_matrix = rho
    with Hierarchy(p) as h:
        h.set_steady_deflation(0)
        st = h.steady_state(ell=ell, tol=1e-10, check=False)
        assert st["status"] == capi.PHI_E_NO_CONVERGENCE and not st["converged"]
        x = h.get_state()
        left = h.apply(x)
        assert np.allclose(h.rho0(), np.eye(n) / n, rtol=0, atol=1e-15)
    # The first tier holds sp Im(c) X_mm 2 / gamma; without it the operator
    # leaves its source terms.  1e-14: a few roundings of values below 10.
    assert np.abs(x.reshape(-1, 2 * n * n)[1:]).max() > 0.05
    assert np.abs(left).max() <= 1e-14 * max(1.0, 16 * np.abs(x).max())
