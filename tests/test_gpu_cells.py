"""The cell list behind the neighbour searches: features and Hamiltonian where
cells are few, open, far apart or unwrapped, against all pairs (the features'
oracle; numpy for the pattern).  Features are FP32 sums of a few dozen terms
below one: 1e-5, as in the oracle test of the periodic cell."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu
EDGE = 7.16 * 1.88973


def _moved(m, box, rng):
    """Atoms carried over by whole periods, either way."""
    k = rng.integers(-2, 3, (m.natoms, 3))
    return m.xyz + k * np.where(np.asarray(box) > 0, box, 0.0)


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 4), (3, 3, 3), (5, 4, 3)])
@pytest.mark.parametrize("open_edges", [(), (2,), (0, 1, 2)])
def test_features_over_cells(gpu, dims, open_edges):
    m = gpu.model_cristobalite(*dims, sigma_ang=0.1, seed=sum(dims))
    box = np.array(dims, float) * EDGE
    box[list(open_edges)] = 0.0
    xyz = _moved(m, box, np.random.default_rng(1))
    ref = MO.features(xyz, m.species, box)
    np.testing.assert_allclose(gpu.mlp_features(xyz, m.species, box), ref, rtol=1e-5, atol=1e-5)


def test_features_of_far_apart_and_single_atoms(gpu):
    xyz = np.array([[0, 0, 0], [3.0, 0, 0], [1e7, 0, 0], [1e7, 3.0, 0], [-4e8, 5, 5]])
    sp = np.array([14, 8, 14, 8, 8], np.int32)
    box = np.zeros(3)
    np.testing.assert_allclose(gpu.mlp_features(xyz, sp, box), MO.features(xyz, sp, box), rtol=1e-5, atol=1e-5)
    assert np.all(gpu.mlp_features(xyz[:1], sp[:1], box) == 0)
    assert np.isnan(gpu.mlp_features(np.where(xyz == 5, np.nan, xyz), sp, box)[0]).any()


@pytest.mark.parametrize("dims,open_edges", [((1, 1, 1), ()), ((2, 1, 3), (2,)), ((3, 2, 2), (0, 1, 2)), ((4, 4, 4), ())])
def test_geometry_over_cells(gpu, dims, open_edges):
    """Density on the device-built H against the same H from all pairs (numpy
    pattern, the host model's blocks where every edge is periodic)."""
    m = gpu.model_cristobalite(*dims, sigma_ang=0.08, seed=3)
    box = np.array(dims, float) * EDGE
    full = box.copy()
    box[list(open_edges)] = 0.0
    xyz = _moved(m, box, np.random.default_rng(2)) if not open_edges else m.xyz
    d = xyz[None] - xyz[:, None]
    d -= np.where(box > 0, box, 1.0) * np.where(box > 0, np.round(d / np.where(box > 0, box, 1.0)), 0.0)
    near = (d ** 2).sum(-1)
    pairs = int(((near < 16) & (near > 0.1)).sum())
    with gpu.Context(M=20, kT=0.1, fp64_small=-1) as c:
        c.set_geometry(xyz, m.species, box)
        r = c.density()
        # tr X^2 counts every stored block; the pattern alone shows in the Coulomb matrix
        V = np.array([c.coulomb_shift(m.q0 + np.eye(m.natoms)[a]) for a in range(0, m.natoms, max(1, m.natoms // 50))])
    step = max(1, m.natoms // 50)
    g = np.where((near < 16) & (near > 0.1), 1.0 / np.sqrt(np.where(near > 0, near, 1.0)), 0.0) + np.eye(m.natoms)
    np.testing.assert_allclose(V, g[::step], rtol=0, atol=1e-12)
    assert pairs > 0 and abs(r["q"].sum() - m.n_electrons) < 1e-6
    if not open_edges and max(dims) > 1:
        with gpu.Context(M=20, kT=0.1, fp64_small=-1) as c:
            c.set_model(gpu.model_cristobalite(*dims, sigma_ang=0.08, seed=3))
            np.testing.assert_allclose(r["q"], c.density()["q"], rtol=0, atol=1e-9)


def test_features_of_an_atom_with_a_crowd(gpu):
    """More near atoms than the list holds: the walk over all atoms."""
    rng = np.random.default_rng(5)
    xyz = rng.uniform(0, 12.0, (400, 3))
    sp = np.where(rng.random(400) < 0.4, 14, 8).astype(np.int32)
    ref = MO.features(xyz, sp, np.zeros(3))
    np.testing.assert_allclose(gpu.mlp_features(xyz, sp, np.zeros(3)), ref, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("rcut", [7.0, 11.0, 60.0])
def test_geometry_with_long_rows(gpu, rcut):
    """Wider cutoffs: rows of about 10, more than 32 and more than 256 neighbours."""
    m = gpu.model_cristobalite(3, 2, 2, sigma_ang=0.08, seed=3)
    d = ((m.xyz[None] - m.xyz[:, None]) ** 2).sum(-1)
    on = (d < rcut ** 2) & (d > 0.1)
    assert {7.0: 8, 11.0: 32, 60.0: 256}[rcut] < on.sum(1).max() + 1
    g = np.where(on, 1.0 / np.sqrt(np.where(d > 0, d, 1.0)), 0.0) + np.eye(m.natoms)
    with gpu.Context(M=20) as c:
        c.set_geometry(m.xyz, m.species, np.zeros(3), rcut_bohr=rcut)
        for a in range(0, m.natoms, 29):
            np.testing.assert_allclose(c.coulomb_shift(m.q0 + np.eye(m.natoms)[a]), g[a], rtol=0, atol=1e-12)
