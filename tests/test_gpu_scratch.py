"""Device memory after calls that took much of it, and after one that could not have it."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def _chain(nb):
    A = sp.kron(sp.diags([np.ones(nb - 1), np.linspace(0, 0.1, nb), np.ones(nb - 1)], [-1, 0, 1]), np.eye(4)).tocsr()
    A.sort_indices()
    return A.indptr, A.indices, A.data, np.repeat(np.arange(nb, dtype=np.int32), 4), nb


def test_out_of_memory_leaves_no_configuration(gpu):
    """The column sums of M = 6000 over one slab of 32768 columns would take
    more than the device has (K x groups x columns x 16 bytes, 402 GB with the
    largest groups, 32 block rows; one allocation, refused at once).  The same
    call again is refused again, and a call that fits gives what a new context
    gives."""
    n = 4 * 8192
    kw = dict(precision=gpu.PREC_FP32, fp32_kernel=4, column_block=n, n_electrons=1.0 * n)
    with gpu.Context(M=6000, **kw) as c, gpu.Context(M=20, **kw) as ref:
        c.set_hamiltonian(*_chain(8192))
        for _ in range(2):
            with pytest.raises(gpu.TbError) as e:
                c.density()
            assert e.value.status == 11, e.value  # TB_ERR_OUT_OF_MEMORY
        c.set_params(M=20, **kw)
        r = c.density()
        ref.set_hamiltonian(*_chain(8192))
        np.testing.assert_array_equal(r["diagP"], ref.density()["diagP"])


def test_stochastic_scratch_is_bounded(gpu):
    """1.6 GB for 4096 probes of 16000 orbitals on a caller's interval go back
    with the call, but for at most 512 MB (and X); the moment of order 0 is the
    sum of the probes' squares, one a deviate, to 5 of its standard deviations."""
    import torch
    with gpu.Context(M=4, n_electrons=8000.0, bounds_lo=-3.0, bounds_hi=3.0) as c:
        c.set_hamiltonian(*_chain(4000))
        c.kpm_dos(n_moments=4, n_random=1, seed=1, npts=8)
        before = torch.cuda.mem_get_info()[0]
        r = c.kpm_dos(n_moments=4, n_random=4096, seed=1, npts=8)
        assert before - torch.cuda.mem_get_info()[0] <= 512 << 20
    n = 16000 * 4096
    assert abs(r["moments"][0] - n) < 5 * np.sqrt(2.0 * n)
