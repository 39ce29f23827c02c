"""Mode rotation of g(Re, q) at the edges of its two forms (registers per entry, a thread per output), FP64, against numpy
in 64 bits: a sum over Rp and one over the modes, every entry within (K + nm + 16) eps of the sum of its terms'
magnitudes."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


@pytest.mark.gpu
@pytest.mark.parametrize("nw,nm,n_el,nq", [(1, 1, 0, 1), (1, 3, 1, 3), (1, 6, 3, 6), (1, 12, 6, 1), (1, 12, 6, 7), (1, 15, 10, 1),
                                           (1, 18, 1, 2), (2, 9, 1, 5), (3, 15, 2, 2), (2, 16, 1, 3)])
def test_modes(nw, nm, n_el, nq):
    import torch

    from epb200 import batched as B
    from epb200 import synth
    from epb200.wannier import WannierObject, to_device

    rng = np.random.default_rng([nw, nm, n_el])
    re, rp = synth.irvec_box(n_el), synth.irvec_box(1)

    def cn(*s):
        return np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s))

    op = cn(nw * nw * nm * len(re), len(rp))
    u, x = cn(nm, nm, nq), np.asfortranarray(rng.random((3, nq)))
    itp = B.get_interpolator(to_device(WannierObject(rp, op, irvec_next=re)))
    guard = torch.full((nq + 1, len(re), nw * nw * nm), 7.0 + 0j, dtype=torch.complex128, device="cuda")
    B.get_eph_RR_to_Rq_batched(guard[:nq], itp, x, B.jl(u))
    got = guard.cpu().numpy()

    def turn(g, w):  # (nb, nm, nr, nq) by (mu, nu, q)
        return np.einsum("bmrq,mnq->bnrq", g.reshape((nw * nw, nm, len(re), nq), order="F"), w)

    ph = np.exp(2j * np.pi * (rp @ x))
    ref = turn(op @ ph, u)
    bar = (len(rp) + nm + 16) * EPS * turn(np.abs(op) @ np.abs(ph), np.abs(u))
    have = got[:nq].transpose(2, 1, 0).reshape(ref.shape, order="F")
    assert (np.abs(have - ref) <= bar).all()
    assert (got[nq] == 7.0).all()
