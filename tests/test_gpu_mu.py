"""The chemical potential's multisection evaluates the Fermi function within
40 kT of a candidate only and takes the nodes below from sums of four; the
charges' coefficients are taken over all nodes, so the charges' sum checks the
count that the search saw: windows wider than the interval, inside it and a
few nodes narrow, mu low, amid and high in the spectrum.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the spectrum's half width is 2: beta_x of 8, 40, 290 (node factors), 3000 and 1e6
# (exponentials; steps of the count in the last bracket), and the step function
@pytest.mark.parametrize("kT", [0.25, 0.05, 0.0068, 0.00066, 2e-6, 0.0])
@pytest.mark.parametrize("fill", [0.05, 0.5, 0.95])
def test_electron_count_of_mu(gpu, kT, fill):
    """The search ends within mu_tol = 1e-9; both counts add the same terms in another order, 1e-12 n."""
    m = gpu.model_cristobalite(1, 1, 1, sigma_ang=0.05, seed=2)
    ne = 2.0 * m.n * fill
    m.q0[:] = ne / m.natoms
    tol = 1e-9 + 1e-12 * m.n
    with gpu.Context(M=64, kT=kT, n_electrons=ne) as c:
        c.set_model(m)
        assert abs(c.density()["q"].sum() - ne) <= tol
    with gpu.Batch([m, m], M=64, kT=kT, scc_max_iter=1) as b:
        for q in b.scc_solve(raise_on_cap=False)["q"]:
            assert abs(q.sum() - ne) <= tol
