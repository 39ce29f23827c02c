"""Graph mode of epb_eph_pass beyond one set of buffers: every call's results are those of the eager pass on its own
arguments, whatever other calls came between."""
import numpy as np
import pytest

from epb200 import synth


def _run(P, dm, xk, xq, out=None, k_batch=4):
    return P.run_eph_over_k_and_q(dm, xk, xq, prec=P.PREC_FP64, k_batch=k_batch, sample_stride=3, out=out)


def _arrays(r):
    from epb200.batched import host

    return [host(t).copy() for t in (r.ek, r.omega, r.g2_sample)]  # g2sum is added up in no fixed order


@pytest.fixture
def graph_mode():
    """A stream of its own (the legacy default stream is never captured) with the default context in graph mode."""
    import torch

    from epb200 import _lib

    with torch.cuda.stream(torch.cuda.Stream()):
        ctx = _lib.default_context()
        ctx.set_graph_mode(True)
        try:
            yield ctx
        finally:
            ctx.set_graph_mode(False)
            torch.cuda.synchronize()


@pytest.mark.gpu
def test_two_sets_of_buffers(graph_mode):
    """A pass captured for one set of buffers is not replayed for another."""
    from epb200 import pipeline as P
    from epb200.batched import jl

    dm = P.DeviceModel(synth.config2_model(seed=3, n_el=1, n_ph=1, nw=5, natom=2))
    points = [(jl(synth.random_kpoints(9, s)), jl(synth.random_kpoints(33, s + 1))) for s in (10, 20)]
    graph_mode.set_graph_mode(False)
    ref = [_arrays(_run(P, dm, *p)) for p in points]
    graph_mode.set_graph_mode(True)
    outs = [None, None]
    for which in (0, 0, 0, 1, 1, 1, 0, 1, 0, 0):
        if outs[which] is not None:
            for t in (outs[which].ek, outs[which].omega, outs[which].g2_sample):
                t.fill_(-1)
        outs[which] = _run(P, dm, *points[which], out=outs[which])
        for a, b in zip(_arrays(outs[which]), ref[which]):
            np.testing.assert_array_equal(a, b)
    dm.close()


def _grow(nw, nm, n_el, nk):
    """Larger calls on the same context: the scratch of the FP64 Fourier sums and of RR -> kR moves."""
    import torch

    from epb200 import batched as B
    from epb200.wannier import WannierObject, to_device

    rng = np.random.default_rng(nk)
    irvec, ir_ep = synth.irvec_box(n_el), synth.irvec_box(1)
    op = rng.standard_normal((nw * nw * nm * len(ir_ep), len(irvec))) + 0j
    obj = to_device(WannierObject(irvec, np.asfortranarray(op), irvec_next=ir_ep))
    x = np.asfortranarray(rng.random((3, nk)))
    itp = B.get_interpolator(obj)
    B.get_fourier_batched(itp, x)
    uks = B.jl(np.repeat(np.eye(nw, dtype=complex)[:, :, None], nk, axis=2))
    B.get_eph_RR_to_kR_batched(B.jl_empty((nw * nw * nm, len(ir_ep), nk), torch.complex128), itp, x, uks)


@pytest.mark.gpu
def test_workspaces_that_move(graph_mode):
    """Larger calls between captured passes move the scratch that the graph has the address of: the pass runs again
    on the new one. Sizes at which the FP64 vertex product keeps its operands in that scratch."""
    from epb200 import pipeline as P
    from epb200.batched import jl

    dm = P.DeviceModel(synth.config2_model(seed=4, n_el=1, n_ph=2, nw=16, natom=4))
    xk, xq = jl(synth.random_kpoints(3, 30)), jl(synth.random_kpoints(4096, 31))
    graph_mode.set_graph_mode(False)
    ref = _arrays(_run(P, dm, xk, xq, k_batch=2))
    graph_mode.set_graph_mode(True)
    out, held = None, []
    for grow in (0, 0, 0, 600, 0, 0, 2500, 0, 0):
        if grow:
            _grow(8, 6, 2, grow)
        held.append(graph_mode.workspace_bytes())
        if out is not None:
            for t in (out.ek, out.omega, out.g2_sample):
                t.fill_(-1)
        out = _run(P, dm, xk, xq, out, k_batch=2)
        for a, b in zip(_arrays(out), ref):
            np.testing.assert_array_equal(a, b)
    assert held[3] > held[2] and held[6] > held[5]  # the calls in between did grow them
    dm.close()


@pytest.mark.gpu
def test_sum_in_a_callers_graph(graph_mode):
    """A large FP64 Fourier sum in a graph that the caller captures uses none of the context's scratch: it replays
    after larger calls have moved that."""
    import torch

    from epb200 import batched as B
    from epb200.wannier import WannierObject, to_device

    rng = np.random.default_rng(1)
    irvec = synth.irvec_box(2)
    op = rng.standard_normal((1500, len(irvec))) + 1j * rng.standard_normal((1500, len(irvec)))
    itp = B.get_interpolator(to_device(WannierObject(irvec, np.asfortranarray(op))))
    x = B.jl(np.asfortranarray(rng.random((3, 3000))))
    out = B.jl_empty((1500, 3000), torch.complex128)
    eager = B.get_fourier_batched(itp, x).clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        B.get_fourier_batched(itp, x, out=out)
    _grow(8, 6, 2, 2500)
    bar = 2 * (len(irvec) + 16) * np.finfo(np.float64).eps * np.abs(op).sum(axis=1).max()
    for _ in range(2):
        out.fill_(-1)
        g.replay()
        assert (out - eager).abs().max().item() <= bar
    del g


@pytest.mark.gpu
def test_not_finite_once(graph_mode):
    """A replay whose points are NaN is done by the FP64 tensor cores; the next one, finite again, has the bits of the
    digit form."""
    import torch

    from epb200 import pipeline as P
    from epb200.batched import jl

    dm = P.DeviceModel(synth.config2_model(seed=5, n_el=1, n_ph=2, nw=16, natom=4))
    xk, xq = jl(synth.random_kpoints(2, 40)), jl(synth.random_kpoints(4096, 41))
    out = None
    for _ in range(3):  # eager, capture, replay
        out = _run(P, dm, xk, xq, out, k_batch=2)
    ref = _arrays(out)
    q = xq.clone()
    xq[5] = np.nan
    out = _run(P, dm, xk, xq, out, k_batch=2)
    assert np.isnan(_arrays(out)[1][:, 5]).any()
    xq.copy_(q)
    for _ in range(2):
        out = _run(P, dm, xk, xq, out, k_batch=2)
        for a, b in zip(_arrays(out), ref):
            np.testing.assert_array_equal(a, b)
    dm.close()
