"""FP64 gauge rotations on q lists long enough for the register kernels (epb_rot64.cu), every number of four-band steps
and of register modes, with tiles that the bands fill partly, below four tiles a q and from four on (operands staged):
sampled q against numpy in 64 bits, every entry within (nw + nm + 16) eps of the sum of its terms' magnitudes."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


def _rotate(g, u, p):
    return np.einsum("imq,inaq,abq->mnbq", u, g, p, optimize=True)


@pytest.mark.gpu
@pytest.mark.parametrize("nw,nbk,nbkq,nm,nq", [
    (1, 1, 1, 1, 205), (4, 4, 4, 4, 1331), (5, 1, 3, 1, 233), (8, 4, 8, 4, 261), (8, 7, 8, 7, 342), (8, 7, 8, 10, 545),
    (8, 7, 8, 14, 618), (9, 1, 4, 1, 204), (12, 4, 7, 4, 230), (11, 7, 11, 8, 222), (11, 8, 11, 10, 203),
    (12, 7, 12, 13, 300), (16, 3, 7, 4, 205), (14, 5, 14, 8, 208), (16, 6, 16, 13, 212), (18, 1, 9, 1, 205),
    (30, 2, 24, 4, 240), (25, 3, 24, 8, 212), (23, 4, 21, 10, 210), (32, 4, 15, 13, 206),
    (9, 9, 9, 1, 252), (10, 10, 10, 4, 228), (10, 9, 9, 7, 228), (11, 9, 11, 10, 238), (10, 9, 10, 13, 230),
    (13, 9, 10, 1, 205), (15, 9, 10, 4, 220), (14, 9, 9, 7, 206), (13, 9, 10, 14, 203), (16, 16, 16, 12, 900),
    (29, 1, 25, 1, 464), (25, 3, 25, 6, 219), (32, 2, 28, 9, 202), (31, 5, 28, 12, 202), (26, 3, 25, 13, 212)])
def test_lists(nw, nbk, nbkq, nm, nq):
    import torch

    from epb200 import batched as B

    gen = torch.Generator(device="cuda").manual_seed(nw * 1000 + nm)

    def cn(*s):
        return torch.randn(s[::-1], dtype=torch.complex128, device="cuda", generator=gen)

    dg, du, dp = cn(nw, nbk, nm, nq), cn(nw, nbkq, nq), cn(nm, nm, nq)
    dw = torch.rand((nq, nm), dtype=torch.float64, device="cuda", generator=gen) + 0.5
    ep = torch.full((nq + 1, nm, nbk, nbkq), 7.0 + 0j, dtype=torch.complex128, device="cuda")
    g2 = torch.full((nq + 1, nm, nbk, nbkq), 7.0, dtype=torch.float64, device="cuda")
    B.eph_apply_rotations(ep[:nq], dg, du, dp, g2_out=g2[:nq], omega=dw)
    qs = np.unique(np.concatenate([[0, 1, nq - 2, nq - 1], np.random.default_rng(nm).integers(0, nq, 12)]))
    g, u, p, w = (B.host(t[torch.from_numpy(qs).cuda()]) for t in (dg, du, dp, dw))
    ref = _rotate(g, u.conj(), p)
    bar = (nw + nm + 16) * EPS * _rotate(np.abs(g), np.abs(u), np.abs(p))
    at = torch.from_numpy(qs).cuda()
    assert (np.abs(B.host(ep[at]) - ref) <= bar).all()
    ref2 = np.abs(ref) ** 2 / (2 * w[None, None])
    bar2 = (2 * np.abs(ref) * bar + bar * bar) / (2 * w[None, None]) + 8 * EPS * ref2
    assert (np.abs(B.host(g2[at]) - ref2) <= bar2).all()
    assert (ep[nq] == 7.0).all() and (g2[nq] == 7.0).all()  # nothing past the last q
    only = torch.full_like(g2, 7.0)
    B.eph_apply_rotations(None, dg, du, dp, g2_out=only[:nq], omega=dw)
    assert torch.equal(only, g2)


@pytest.mark.gpu
@pytest.mark.parametrize("over", ["g", "ukq", "uph"])
def test_over_an_input(over):
    """ep written over an input whose blocks of a q are as large as its own: every q is read before it is written."""
    import torch

    from epb200 import batched as B

    nw, nbk, nbkq, nm, nq = {"g": (10, 5, 10, 6, 2000), "ukq": (16, 4, 16, 4, 6000), "uph": (9, 1, 9, 9, 3000)}[over]
    rng = np.random.default_rng(nq)

    def cn(*s):
        return B.jl(np.asfortranarray(rng.standard_normal(s) + 1j * rng.standard_normal(s)))

    args = {"g": cn(nw, nbk, nm, nq), "ukq": cn(nw, nbkq, nq), "uph": cn(nm, nm, nq)}
    g, u, p = (B.host(args[k]).copy() for k in ("g", "ukq", "uph"))
    ref = _rotate(g, u.conj(), p)
    bar = (nw + nm + 16) * EPS * _rotate(np.abs(g), np.abs(u), np.abs(p))
    ep = args[over].view(nq, nm, nbk, nbkq)
    B.eph_apply_rotations(ep, args["g"], args["ukq"], args["uph"])
    assert (np.abs(B.host(ep) - ref) <= bar).all()
