"""The stochastic density over several slabs of probes.

A slab of fixed-point probes is scaled by a power of two of its own largest
entry, so slabs whose largest entries lie on both sides of a power of two must
still count alike.  Tolerances: both sides draw the same probes and run the
same recurrence in 64 bits, off by some 1e-15 an order; 1e-9 (of the largest
entry where T_k grows past one) holds both with room; a wrong scale of one slab
shows at 1e-2.
"""
import numpy as np
import pytest

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
