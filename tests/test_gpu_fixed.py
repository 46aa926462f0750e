"""The FP64 form's fixed-point recurrence at the sizes where it can go wrong.

Tolerances: the oracle's own FP64 recurrence is off by a few 1e-16 times the
order (6e-15 at M = 6000), so 1e-12 on a diagonal moment's sum and on diagP
holds both sides with room; a lost carry or a wrong limb shows at 1e-9 (2^-30).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _random_h(nb, per_row, seed):
    """A symmetric 4x4-block matrix with about per_row blocks a row."""
    import scipy.sparse as sp
    r = np.random.default_rng(seed)
    A = np.zeros((4 * nb, 4 * nb))
    for I in range(nb):
        for J in {I} | set(r.choice(nb, min(nb, per_row) // 2, replace=False)):
            A[4 * I:4 * I + 4, 4 * J:4 * J + 4] += r.normal(size=(4, 4))
    H = sp.csr_matrix((A + A.T) / 2)
    H.sort_indices()
    return H


# 1 atom (one block, 4 of 64 columns); 17 and 33 atoms (ragged warps and
# column groups); rows of about 30, 53 and 67 blocks (no, one and two flushes);
# 80 sparse rows with two slabs
@pytest.mark.parametrize("nb,per_row,B,pad", [(1, 2, 0, 0.05), (17, 6, 0, 0.0), (33, 4, 0, 0.0), (40, 80, 0, 0.0),
                                              (70, 140, 0, 0.01),
                                              (90, 180, 0, 0.0), (80, 8, 128, 0.0)])
def test_fixed_point_matches_oracle(gpu, nb, per_row, B, pad):
    H = _random_h(nb, per_row, nb)
    M, ne = 60, 4.0 * nb
    o = O.model_from_csr(H.indptr, H.indices, H.data, nb)
    lo, hi = O.gershgorin(o)
    a, b = 0.5 * (hi - lo) * (1 + pad), 0.5 * (hi + lo)
    d = O.exact_moments(o, a, b, M + 1)
    with gpu.Context(M=M, kT=0.02 * (hi - lo), n_electrons=ne, column_block=B, spectral_pad=pad) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.density()
    np.testing.assert_allclose(r["moments"], d[:M + 1].sum(axis=1), rtol=0, atol=1e-12 * 4 * nb)
    assert abs(r["q"].sum() - ne) < 1e-8
    if pad == 0.0:
        ref = O.density(o, O.kpe_params(M=M, kT=0.02 * (hi - lo), n_elec=ne))
        np.testing.assert_allclose(r["diagP"], ref["diagP"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("nr", [1, 32, 33, 130])
def test_probe_moments_match_oracle(gpu, nr):
    """Probe slabs of 32 and of multiples of 64 columns, several slabs; moments
    are sums of nr * n products, 1e-12 of each."""
    H = _random_h(33, 5, 3)
    o = O.model_from_csr(H.indptr, H.indices, H.data, 33)
    with gpu.Context(M=20, n_electrons=66.0) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(33, dtype=np.int32), 4), 33)
        r = c.kpm_dos(n_moments=41, n_random=nr, seed=7, npts=30)
    a, b = r["report"]["a"], r["report"]["b"]
    mom, e, dos = O.kpm_dos(o, a, b, nmom=41, n_random=nr, seed=7, npts=30)[:3]
    np.testing.assert_allclose(r["moments"], mom, rtol=0, atol=1e-12 * nr * 132)
    np.testing.assert_allclose(r["dos"], dos, rtol=0, atol=1e-11 * nr * 132)


@pytest.mark.parametrize("npts,ne", [(3, 132.0), (40, 66.0)])
def test_density_outside_the_interval_starts_again_in_fp64(gpu, npts, ne):
    """A chain fills its Gershgorin interval; refined from three DOS nodes, the
    interval leaves the band's ends outside, T_k x passes the fixed range and
    the pass is made again in FP64 (diagP runs far past one): as the oracle, to
    rounding.  With forty nodes it stays in range."""
    import scipy.sparse as sp
    nb = 33
    A = sp.kron(sp.diags([np.ones(nb - 1), np.linspace(0, 0.1, nb), np.ones(nb - 1)], [-1, 0, 1]), np.eye(4)).tocsr()
    A.sort_indices()
    o = O.model_from_csr(A.indptr, A.indices, A.data, nb)
    p = O.kpe_params(M=40, kT=0.0, n_elec=ne)
    with gpu.Context(M=40, kT=0.0, n_electrons=ne) as c:
        c.set_hamiltonian(A.indptr, A.indices, A.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.density_stochastic(n_probes=6, seed=2, dos_moments=30, dos_points=npts)
    ref = O.density_stochastic(o, p, n_random=6, seed=2, dos_moments=30, dos_points=npts)
    s = np.abs(ref["diagP"]).max()
    assert (s > 10) == (npts == 3)
    np.testing.assert_allclose(r["diagP"], ref["diagP"], rtol=0, atol=1e-9 * max(1.0, s))
