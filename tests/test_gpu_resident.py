"""The column-resident recurrence (T_k on chip, one launch for all steps) at
the edges of its chunks of 32 block rows and of its shared memory.

Its T_k is the slab kernels' to the bit; only the column sums are added in
another order, as pairs of ~44 bits, so a diagonal moment differs by a few
2^-44 at most: 1e-12 an orbital on the traces, with room.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band_h(nb, reach, seed):
    """Block-banded symmetric H: row I meets I +- 1 .. reach, a third of the rows one more far away."""
    import scipy.sparse as sp
    r = np.random.default_rng(seed)
    I, J = [], []
    for a in range(nb):
        for b in [a] + [a + d for d in range(1, reach + 1) if a + d < nb] + ([int(r.integers(nb))] if a % 3 == 0 else []):
            I.append(a)
            J.append(b)
    B = sp.bsr_matrix((r.normal(size=(len(I), 4, 4)), np.array(J), np.searchsorted(I, np.arange(nb + 1))),
                      shape=(4 * nb, 4 * nb)).tocsr()
    H = ((B + B.T) / 2).tocsr()
    H.sum_duplicates()
    H.sort_indices()
    return H


def _density(gpu, H, **kw):
    nb = H.shape[0] // 4
    with gpu.Context(M=50, kT=0.2, n_electrons=4.0 * nb, fp64_small=-1, **kw) as c:
        c.set_hamiltonian(H.indptr, H.indices, H.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb)
        return c.density()


# one row; a chunk less, exactly and more; several; the last size that fits
@pytest.mark.parametrize("nb,reach", [(1, 1), (31, 2), (32, 1), (33, 5), (100, 40), (257, 3), (1792, 1)])
def test_resident_equals_slab_kernels(gpu, nb, reach):
    H = _band_h(nb, reach, nb)
    a = _density(gpu, H, precision=gpu.PREC_FP32, fp32_kernel=gpu.FP32_PERSISTENT)
    b = _density(gpu, H, precision=gpu.PREC_FP32, fp32_kernel=gpu.FP32_STAGED)
    assert a["report"]["step_kernel"] == gpu.FP32_PERSISTENT
    assert b["report"]["step_kernel"] == gpu.FP32_STAGED
    np.testing.assert_allclose(a["moments"], b["moments"], rtol=0, atol=1e-12 * 4 * nb)
    np.testing.assert_allclose(a["diagP"], b["diagP"], rtol=0, atol=1e-9)


@pytest.mark.parametrize("nb", [33, 257, 1792, 1793])
def test_fixed_point_resident_equals_slabs(gpu, nb):
    """Same integers either way, added in another order: rounding of the last place."""
    H = _band_h(nb, 2, nb)
    a = _density(gpu, H, precision=gpu.PREC_FP64)
    b = _density(gpu, H, precision=gpu.PREC_FP64, column_block=128)
    np.testing.assert_allclose(a["moments"], b["moments"], rtol=0, atol=1e-14 * 4 * nb)


# a lane takes one row of a block up to three chunks, all four beyond
@pytest.mark.parametrize("nb,reach", [(1, 1), (32, 3), (64, 40), (96, 2), (97, 2)])
def test_fixed_point_resident_by_rows_of_a_block(gpu, nb, reach):
    """As above: the same integers."""
    H = _band_h(nb, reach, nb)
    a = _density(gpu, H, precision=gpu.PREC_FP64)
    b = _density(gpu, H, precision=gpu.PREC_FP64, column_block=128)
    np.testing.assert_allclose(a["moments"], b["moments"], rtol=0, atol=1e-14 * 4 * nb)


# the first size that AUTO steps so and the first that does not fit on chip;
# rows that are no multiple of 16 or of a row group, runs of one chunk and of
# four; long-range links (many mirrored rows)
@pytest.mark.parametrize("nb,reach", [(897, 2), (1441, 1), (1793, 1), (1800, 4), (2047, 2)])
def test_symmetric_half_is_as_exact_as_the_whole_slab(gpu, nb, reach):
    """From there on AUTO steps the symmetric half of one slab: T_k then rounds
    differently, by as much.  Against the FP64 form, its errors are those of
    the whole slab (within half as much again), and both within the FP32 bars
    of the oracle tests."""
    H = _band_h(nb, reach, nb)
    ref = _density(gpu, H, precision=gpu.PREC_FP64)
    half = _density(gpu, H, precision=gpu.PREC_FP32)
    whole = _density(gpu, H, precision=gpu.PREC_FP32, fp32_kernel=gpu.FP32_PIPELINED_STEP)
    again = _density(gpu, H, precision=gpu.PREC_FP32)
    assert half["report"]["step_kernel"] == gpu.FP32_PIPELINED_STEP
    assert half["report"]["column_block"] == -(-4 * nb // 64) * 64
    np.testing.assert_array_equal(half["moments"], again["moments"])
    for key, bar in (("q", 1e-6), ("diagP", 1e-6)):
        e = {n: np.abs(r[key] - ref[key]) for n, r in (("half", half), ("whole", whole))}
        assert e["half"].max() < bar
        assert np.sqrt((e["half"] ** 2).mean()) <= 1.5 * np.sqrt((e["whole"] ** 2).mean()), key
    np.testing.assert_allclose(half["moments"], ref["moments"], rtol=0, atol=2e-5 * 4 * nb)


def test_batch_mixes_resident_and_slab_structures(gpu):
    """Structures of every class beside one that steps on slabs: each as when solved alone."""
    M = 40
    models = [gpu.model_cristobalite(*d, sigma_ang=0.05, seed=5 + i)
              for i, d in enumerate([(5, 4, 4), (1, 1, 2), (3, 3, 3), (4, 4, 3), (2, 2, 3)])]
    with gpu.Batch(models, M=M, kT=0.05, fp64_small=-1) as b:
        r = b.scc_solve()
    for i, m in enumerate(models):
        with gpu.Context(M=M, kT=0.05, precision=gpu.PREC_FP32, fp64_small=-1) as c:
            c.set_model(m)
            s = c.scc_solve()
        assert abs(int(r["iters"][i]) - s["iters"]) <= 1
        assert np.abs(r["q"][i] - s["q"]).max() < 1e-6


def test_chained_steps_in_a_graph(gpu):
    """The steps of the symmetric half overlap their launches; captured or not, the same numbers come out."""
    m = gpu.model_cristobalite(5, 4, 2, sigma_ang=0.05, seed=3)
    out = []
    for no_graphs in (0, 1):
        with gpu.Context(M=40, kT=0.05, precision=gpu.PREC_FP32, fp64_small=-1, no_graphs=no_graphs) as c:
            c.set_model(m)
            out.append(c.scc_solve())
    assert out[0]["report"]["step_kernel"] == gpu.FP32_PIPELINED_STEP
    assert out[0]["iters"] == out[1]["iters"]
    np.testing.assert_array_equal(out[0]["q"], out[1]["q"])
