"""The stochastic density over several slabs of probes, and with an entry of X
far outside the refined interval.

A slab of fixed-point probes is scaled by a power of two of its own largest
entry, so slabs whose largest entries lie on both sides of a power of two must
still count alike.  Tolerances: both sides draw the same probes and run the
same recurrence in 64 bits, off by some 1e-15 an order; 1e-9 (of the largest
entry where T_k grows past one) holds both with room, a wrong scale of one slab
shows at 1e-2.
"""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle as O
from test_gpu_fixed import _random_h

pytestmark = pytest.mark.gpu


def _shift(n, seed, t0, t1):
    """The power of two that brings probes t0 .. t1 - 1 below a quarter."""
    return int(np.ceil(np.log2(4 * max(abs(O.gauss(seed, t * n + i)) for t in range(t0, t1) for i in range(n)))))


# on the caller's interval slabs of 256: a full one and a rest, shifts up and
# down; on Gershgorin's the probes' share of L2, two of 576, and three; alike
@pytest.mark.parametrize("nb,nr,seed,bounds,slabs", [
    (36, 300, 2, True, [0, 256, 300]), (36, 300, 5, True, [0, 256, 300]), (36, 513, 4, True, [0, 256, 512, 513]),
    (9, 1100, 2, False, [0, 576, 1100]), (9, 2050, 2, False, [0, 704, 1408, 2050]),
    (9, 1100, 4, False, [0, 576, 1100])])
def test_probe_slabs_count_alike(gpu, nb, nr, seed, bounds, slabs):
    H = _random_h(nb, 4, nb)
    n = 4 * nb
    shifts = [_shift(n, seed + 1, a, b) for a, b in zip(slabs, slabs[1:])]
    assert (len(set(shifts)) > 1) == (seed != 4 or bounds)
    o = O.model_from_csr(H.indptr, H.indices, H.data, nb)
    lo, hi = O.gershgorin(o)
    ref = O.density_stochastic(o, O.kpe_params(M=30, kT=0.0, n_elec=4.0 * nb), n_random=nr, seed=seed, dos_moments=40,
                               dos_points=100)
    own = dict(bounds_lo=lo, bounds_hi=hi) if bounds else {}
    with gpu.Context(M=30, kT=0.0, n_electrons=4.0 * nb, **own) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.density_stochastic(n_probes=nr, seed=seed, dos_moments=40, dos_points=100)
    s = max(1.0, np.abs(ref["diagP"]).max())
    np.testing.assert_allclose(r["diagP"], ref["diagP"], rtol=0, atol=1e-9 * s)
    np.testing.assert_allclose(r["q"], ref["q"], rtol=0, atol=8e-9 * s)


@pytest.mark.parametrize("level", [4.2, 5.0, 6.2])
def test_level_far_outside_the_refined_interval(gpu, level):
    """A level of its own that the one probe hardly sees (its deviate is
    -0.014): the DOS leaves it out of the refined interval, 1.8 to 2.6 half
    widths from its centre, and T_k grows there as in FP64."""
    nb, seed = 33, 34
    A = sp.lil_matrix((4 * nb, 4 * nb))
    chain = sp.diags([np.ones(nb - 2), np.linspace(0, 0.1, nb - 1), np.ones(nb - 2)], [-1, 0, 1])
    A[:4 * nb - 4, :4 * nb - 4] = sp.kron(chain, np.eye(4))
    A[4 * nb - 4, 4 * nb - 4] = level
    for i in range(4 * nb - 3, 4 * nb):
        A[i, i] = 0.05
    A = A.tocsr()
    A.sort_indices()
    o = O.model_from_csr(A.indptr, A.indices, A.data, nb)
    ref = O.density_stochastic(o, O.kpe_params(M=12, kT=0.0, n_elec=4.0 * nb, pad=0.3), n_random=1, seed=seed,
                               dos_moments=200, dos_points=400)
    x = (level - ref["b"]) / ref["a"]
    assert 1.7 < x < 2.9 and (x > 1.9) == (level > 4.2)
    with gpu.Context(M=12, kT=0.0, n_electrons=4.0 * nb, spectral_pad=0.3) as c:
        c.set_hamiltonian(A.indptr, A.indices, A.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.density_stochastic(n_probes=1, seed=seed, dos_moments=200, dos_points=400)
    s = np.abs(ref["diagP"]).max()
    assert s > 10
    np.testing.assert_allclose(r["diagP"], ref["diagP"], rtol=0, atol=1e-9 * s)


@pytest.mark.parametrize("nr", [1100, 2050])
def test_moments_over_slabs(gpu, nr):
    """Two and three slabs of moments: sums of nr n products, 1e-12 of each."""
    nb = 9
    H = _random_h(nb, 4, nb)
    o = O.model_from_csr(H.indptr, H.indices, H.data, nb)
    with gpu.Context(M=20, n_electrons=4.0 * nb) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.kpm_dos(n_moments=41, n_random=nr, seed=2, npts=30)
    a, b = r["report"]["a"], r["report"]["b"]
    mom, e, dos = O.kpm_dos(o, a, b, nmom=41, n_random=nr, seed=2, npts=30)[:3]
    np.testing.assert_allclose(r["moments"], mom, rtol=0, atol=1e-12 * nr * 4 * nb)
    np.testing.assert_allclose(r["dos"], dos, rtol=0, atol=1e-11 * nr * 4 * nb)
