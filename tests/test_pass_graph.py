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
