"""Cutoffs so small that an edge holds more of them than a double counts."""
import pytest

pytestmark = pytest.mark.gpu


# open and periodic edges; 1e-308 and the smallest double: span / cutoff is infinite
@pytest.mark.parametrize("box", [[0.0, 0.0, 0.0], None])
@pytest.mark.parametrize("rcut", [1e-300, 1e-308, 5e-324])
def test_tiny_cutoff_finds_no_neighbour(gpu, rcut, box):
    from largetb_gb300 import learned
    m = gpu.model_cristobalite(1, 1, 1, sigma_ang=0.05, seed=3)
    box = box or learned.cell_box((1, 1, 1))
    with gpu.Context(M=20) as c:
        c.set_geometry(m.xyz, m.species, box, rcut_bohr=0.1)  # atoms are further apart
        alone = c.gershgorin()
        c.set_geometry(m.xyz, m.species, box, rcut_bohr=rcut)
        assert c.gershgorin() == alone
