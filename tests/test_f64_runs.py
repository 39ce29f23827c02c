"""Large FP64 sums whose digit planes are packed in several runs of rows, and of rows and columns."""
import numpy as np
import pytest

from oracle import epb_oracle as O

EPS = np.finfo(np.float64).eps


@pytest.mark.gpu
@pytest.mark.parametrize("ndata,n_el,nk,held", [(40001, 4, 150, 600), (5001, 6, 9001, 1200)])
def test_runs(ndata, n_el, nk, held):
    """Entries within (K + 16) eps of the sum of their row's magnitudes; the context holds no more than the runs (`held`
    MB), and more than none (so that this is the digit form)."""
    import torch

    from epb200 import _lib, synth
    from epb200 import batched as B

    rng = np.random.default_rng(ndata)
    irvec = synth.irvec_box(n_el)
    g = torch.Generator(device="cuda").manual_seed(ndata)
    op = torch.randn((len(irvec), ndata), dtype=torch.complex128, device="cuda", generator=g)
    x = np.asfortranarray(rng.random((3, nk)))
    ctx = _lib.Context(0)
    rset = _lib.RSet(ctx, irvec)
    out = torch.full((nk + 1, ndata), 7.0 + 0j, dtype=torch.complex128, device="cuda")
    dx = B.jl(x)
    _lib.check(_lib.lib().epb_fourier(ctx.h, op.data_ptr(), ndata, ndata, rset.h, dx.data_ptr(), nk, out.data_ptr(), 0))
    cols = np.unique(np.concatenate([rng.integers(0, nk, 20), [0, 127, 128, nk - 1]]))
    got = out[torch.from_numpy(cols).cuda()].cpu().numpy().T
    host = np.asfortranarray(op.cpu().numpy().T)
    ref = O.fourier_batched(host, ndata, irvec, np.asfortranarray(x[:, cols]))
    bar = (len(irvec) + 16) * EPS * np.abs(host).sum(axis=1)
    assert (np.abs(got - ref) <= bar[:, None]).all()
    assert (out[nk] == 7.0).all()
    assert 50e6 < ctx.workspace_bytes() < held * 1e6
    rset.close()
    ctx.close()
