"""Column sums of the FP32 recurrence: every addition keeps its rounding error.

X is exact in FP32, and so is every sum of the four products that one lane adds
in plain FP32: entries of 1/8 and of 2^-16, whose squares are 26 bits apart, at
the same place of 64-column chunks (one lane sees them one after the other).
<T_1,T_1> is then exact if the sums are; mu_2 = 2 |X|^2 - n sums n values of
about one in FP64, to 1e-11, and 1e-10 is a quarter of one small product's share
(4.7e-10).
"""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _matrix(nb, step):
    """Every `step`-th atom coupled to nine atoms, one a chunk, on its left; a
    level at +2 and one at -2 make Gershgorin's interval [-2, 2]."""
    n, reach = 4 * nb, 9
    r, c, v = [n - 1, n - 2], [n - 1, n - 2], [2.0, -2.0]
    for A in range(16 * reach + 37, nb - 1, step):
        for q in range(4):
            for m in range(reach):
                i, j = 4 * A + q, 4 * (16 * (A // 16 - reach + m) + A % 16)
                r += [i, j]
                c += [j, i]
                v += [0.25 if m == 0 else 2.0 ** -15] * 2
    H = sp.coo_matrix((v, (r, c)), shape=(n, n)).tocsr()
    H.sort_indices()
    assert abs(H).sum(axis=1).max() == 2.0
    return H


# groups of 28 block rows (three a warp) and of 24, runs of four chunks and of
# eight; on the caller's interval; over the whole slab
@pytest.mark.parametrize("kw", [{}, dict(bounds_lo=-2.0, bounds_hi=2.0), dict(fp32_kernel=4, column_block=0)])
@pytest.mark.parametrize("nb,step", [(920, 97), (1280, 41), (2240, 41)])
def test_sums_keep_their_errors(gpu, nb, step, kw):
    H = _matrix(nb, step)
    n = 4 * nb
    if kw.get("fp32_kernel"):
        kw = dict(kw, column_block=(n + 127) // 128 * 128)
    with gpu.Context(M=4, precision=gpu.PREC_FP32, kT=0.5, n_electrons=1.0 * n, **kw) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        r = c.density()
    assert r["report"]["step_kernel"] == 4 and r["report"]["column_block"] >= n
    exact = 2 * ((H.data / 2) ** 2).sum() - n
    assert abs(r["moments"][2] - exact) < 1e-10
