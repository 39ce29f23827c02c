"""FP64 states of matrices with a NaN or infinity, anywhere in the upper triangle: every energy and vector entry is NaN
(none is left as it was), and the other matrices of the batch keep theirs."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3, 4, 7, 8, 11, 12, 16, 17, 32, 40, 64])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_eigen(n, bad):
    import torch

    from epb200 import _lib
    from epb200 import batched as B

    rng = np.random.default_rng(n)
    hs = rng.standard_normal((7, n, n)) + 1j * rng.standard_normal((7, n, n))
    hs = hs + hs.conj().transpose(0, 2, 1)
    given = hs.copy()
    for k, (i, j) in {1: (0, n - 1), 4: (n - 1, n - 1), 5: (n // 2, n - 1)}.items():
        given[k, i, j] = bad
    hit = np.array([k in (1, 4, 5) for k in range(7)])
    a = B.jl(np.asfortranarray(given.transpose(1, 2, 0)))
    e = torch.full((7, n), 5.0, dtype=torch.float64, device="cuda")
    st = _lib.lib().epb_eigh_batched(B._ctx().h, a.data_ptr(), n, 7, e.data_ptr(), b"V", 0)
    assert st in (_lib.EPB_OK, _lib.EPB_ERR_NOCONVERGE)
    e, v = e.cpu().numpy(), B.host(a).transpose(2, 0, 1)
    assert np.isnan(e[hit]).all() and np.isnan(v[hit]).all()
    for k in np.flatnonzero(~hit):
        bar = 40 * n * EPS
        norm = np.linalg.norm(hs[k])
        assert np.abs(e[k] - np.linalg.eigvalsh(hs[k])).max() <= bar * norm
        assert np.abs(hs[k] @ v[k] - v[k] * e[k]).max() <= bar * norm
