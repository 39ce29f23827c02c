"""Eigenvalues alone (tridiagonal reduction and bisection) of matrices that fall into blocks, where off-diagonals of the
tridiagonal are zero and bisection points hit levels exactly: against LAPACK. Reduction and bisection are each good to a
few eps of the norm per step, n steps: 10 n eps of the norm. The mixed form of H(k) has 16 bits and more of its entries'
scale three times over: 1e-5 of the norm."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps
ORDERS = [1, 2, 3, 4, 7, 8, 9, 12, 15, 16, 17, 24, 31, 32]


def _matrices(n):
    """Hermitian matrices of order n, each also with its rows (and columns) in another order."""
    rng = np.random.default_rng(n)
    dimers = np.zeros((n, n), dtype=complex)  # one level at 0 (two of them at even orders), then pairs at -1 and 1
    for i in range(1, n - 1, 2):
        dimers[i, i + 1] = dimers[i + 1, i] = 1
    blocks = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    blocks = blocks + blocks.conj().T
    blocks[: n // 2, n // 2:] = blocks[n // 2:, : n // 2] = 0
    chain = np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1) + 0j  # symmetric levels
    gapped = np.diag(np.append(np.arange(1.0, n), n + 1)) + 0j
    out = [np.diag(np.arange(n)), np.diag(np.arange(n) % 3), np.diag(np.arange(n) - n // 2), dimers, dimers[::-1, ::-1],
           blocks, chain, gapped, np.zeros((n, n)), np.eye(n), 1e-3 * dimers + np.diag(np.arange(n) % 2)]
    out += [np.diag(rng.integers(-4, 5, n)) for _ in range(8)]
    out = [np.asarray(h, dtype=complex) for h in out]
    for h in list(out):
        p = rng.permutation(n)
        out.append(h[np.ix_(p, p)])
    return np.stack(out)


def _worst(e, hs):
    """Largest deviation from LAPACK in norms of the matrix."""
    ref = np.linalg.eigvalsh(hs)
    norm = np.maximum(np.linalg.norm(hs, axis=(1, 2)), 1e-300)
    return (np.abs(e - ref).max(axis=1) / norm).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", ORDERS)
def test_eigvals(n):
    from epb200 import batched as B

    hs = _matrices(n)
    e = B.host(B.eigvals_batched(B.jl(np.asfortranarray(hs.transpose(1, 2, 0))))).T
    assert _worst(e, hs) <= 10 * n * EPS


@pytest.mark.gpu
@pytest.mark.parametrize("n", ORDERS)
def test_states_and_bands(n):
    """The same as H(R = 0) of a model: get_el_eigen_valueonly_batched, and epb_bands_eigvals in both precisions."""
    from epb200 import batched as B
    from epb200 import learned as L
    from epb200.wannier import WannierObject, to_device

    x = np.zeros((3, 2))
    for h in _matrices(n):
        obj = WannierObject(np.zeros((1, 3), dtype=np.int64), np.asfortranarray(h.reshape(-1, 1, order="F")))
        got = B.host(B.get_el_eigen_valueonly_batched(B.get_interpolator(to_device(obj)), x)).T
        assert _worst(got, np.stack([h, h])) <= 10 * n * EPS
        bands = L.BandModel(obj)
        assert _worst(B.host(bands.eigvals(x)).T, np.stack([h, h])) <= 10 * n * EPS
        assert _worst(B.host(bands.eigvals(x, prec=L.PREC_MIXED)).T, np.stack([h, h])) <= 1e-5
        bands.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 5, 8, 11, 16, 17, 32])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite(n, bad):
    """A matrix with a NaN or infinity gets no energies, wherever the entry is; its neighbours in the batch keep
    theirs, at any scale whose squares a double holds."""
    from epb200 import batched as B

    rng = np.random.default_rng(n)
    hs = rng.standard_normal((9, n, n)) + 1j * rng.standard_normal((9, n, n))
    hs = hs + hs.conj().transpose(0, 2, 1)
    hs[0] = np.diag(np.arange(n)) + 1e-155 * hs[0]  # columns whose squared length has no reciprocal
    hs[1] *= 1e-140
    hs[3] *= 1e140
    given = hs.copy()
    for k, (i, j) in {2: (0, n - 1), 4: (0, 0), 6: (n - 1, n - 1), 7: (n // 2, n - 1)}.items():
        given[k, i, j] = bad
    hit = np.array([k in (2, 4, 6, 7) for k in range(9)])
    e = B.host(B.eigvals_batched(B.jl(np.asfortranarray(given.transpose(1, 2, 0))))).T
    assert np.isnan(e[hit]).all()
    assert _worst(e[~hit], hs[~hit]) <= 10 * n * EPS
    tiny = np.asfortranarray((1e-170 * hs[5:6]).transpose(1, 2, 0))  # squares underflow: at least of its own size
    e = B.host(B.eigvals_batched(B.jl(tiny)))
    assert np.isfinite(e).all() and np.abs(e).max() <= 2 * n * np.abs(tiny).max()
