"""The matrix form of the digit product (kR -> kq, whose second factor the caller passes): columns as flat as a phase go
through the digits, others to the FP64 tensor cores, and either way an entry is off by no more than rounding on the
scale of its own terms."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


def _product(a, b, nw, nm):
    """a b by get_eph_kR_to_kq_batched with identity rotations (which add exact zeros)."""
    import torch

    from epb200 import batched as B

    nq = b.shape[1]
    nbk = a.shape[0] // (nw * nm)
    eye = [B.jl(np.repeat(np.eye(n, dtype=complex)[:, :, None], nq, axis=2)) for n in (nm, nw)]
    ep = B.jl_empty((nw, nbk, nm, nq), torch.complex128)
    B.get_eph_kR_to_kq_batched(ep, B.jl(np.asfortranarray(a)), B.jl(np.asfortranarray(b)), eye[0], eye[1])
    return B.host(ep).reshape(a.shape[0], nq, order="F")


def _cn(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0, 3, 18])
def test_graded(spread):
    """Rows and columns whose entries lie over 2 * spread decades, in opposite orders: the largest products are where
    neither factor is largest. And a column that is zero in the place of a row's largest entry."""
    nw, nm, K, nq = 16, 6, 125, 6000
    rng = np.random.default_rng(spread)
    a, b = _cn(rng, nw * nw * nm, K), np.exp(2j * np.pi * rng.random((K, nq)))
    grade = 10.0 ** np.linspace(spread, -spread, K)
    a = a * grade
    b = b / grade[:, None]
    a[7] = np.where(np.arange(K) == 0, 1.0, 1e-18)
    b[0, ::2] = 0
    bar = (K + 16) * EPS * np.abs(a) @ np.abs(b)
    assert (np.abs(_product(a, b, nw, nm) - a @ b) <= bar).all()


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [None, "row", "column"])
def test_phases(bad):
    """Phases, rows over many decades, with and without an infinity: every output that it does not reach keeps its
    bound."""
    nw, nm, K, nq = 16, 6, 125, 6000
    rng = np.random.default_rng(5)
    a = _cn(rng, nw * nw * nm, K) * 10.0 ** rng.uniform(-9, 9, (nw * nw * nm, 1))
    b = np.exp(2j * np.pi * rng.random((K, nq)))
    bar, ref = (K + 16) * EPS * np.abs(a).sum(axis=1, keepdims=True), a @ b
    live = np.ones(ref.shape, bool)
    if bad == "row":
        a[40, 3] = np.inf  # the identity rotations add 0 * inf to the rows of its column, and of its modes
        live = live.reshape(nw, nw, nm, nq, order="F")
        live[:, 40 // nw] = False
        live = live.reshape(ref.shape, order="F")
    elif bad == "column":
        b[3, 40] = np.nan
        live[:, 40] = False
    got = _product(a, b, nw, nm)
    assert ((np.abs(got - ref) <= bar) | ~live).all()
    assert np.isfinite(got[live]).all()
    if bad:
        assert not np.isfinite(got[40, 40])


@pytest.mark.gpu
def test_long_sums_at_full_scale():
    """3375 terms, all of them as large as the digits' scale allows, against extended precision. Left out are digit pairs
    of 2^-54.3 in rms per real product, and operands are rounded to 2^-55: errors of random sign over 2 K products, held
    to six standard deviations, and the rounding of the result."""
    nw, nm, K, nq = 8, 3, 3375, 4000
    rng = np.random.default_rng(9)
    full = 0.9975  # of a power of two: seven balanced digits hold 0.996, so the scale is a bit short of it
    a = full * (rng.choice([-1.0, 1.0], (nw * nw * nm, K)) + 1j * rng.choice([-1.0, 1.0], (nw * nw * nm, K)))
    a -= 0.02 * rng.random(a.shape) * (a.real > 0) + 0.02j * rng.random(a.shape) * (a.imag > 0)
    b = full * rng.choice([-1.0, 1.0], (K, nq)) * (1 - 0.02 * rng.random((K, nq))) \
        + 1j * full * rng.choice([-1.0, 1.0], (K, nq)) * (1 - 0.02 * rng.random((K, nq)))
    cols = np.sort(rng.choice(nq, 24, replace=False))
    ref = a.astype(np.clongdouble) @ b[:, cols].astype(np.clongdouble)
    err = _product(a, b, nw, nm)[:, cols] - ref
    bar = 6 * np.sqrt(2 * K) * (2.0 ** -54.3 + 2.0 ** -55)
    for e, r in ((err.real, ref.real), (err.imag, ref.imag)):
        assert (np.abs(e) <= bar + EPS * np.abs(r)).all()
