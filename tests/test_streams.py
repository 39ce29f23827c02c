"""Calls of one context on two streams without a wait of the host in between: what large FP64 calls keep in the context
between their kernels (operand planes, work counters) serves one after the other."""
import numpy as np
import pytest


@pytest.mark.gpu
def test_large_sums():
    """FP64 Fourier sums of different operands and sizes, alternating between two streams: the bits of the serial
    results. The second size moves the scratch of the first."""
    import torch

    from epb200 import batched as B
    from epb200 import synth
    from epb200.wannier import WannierObject, to_device

    rng = np.random.default_rng(2)
    irvec = synth.irvec_box(2)
    calls = []
    for ndata, nk in ((1500, 3000), (1100, 4100), (2600, 6000)):
        op = rng.standard_normal((ndata, len(irvec))) + 1j * rng.standard_normal((ndata, len(irvec)))
        itp = B.get_interpolator(to_device(WannierObject(irvec, np.asfortranarray(op))))
        x = B.jl(np.asfortranarray(rng.random((3, nk))))
        calls.append((itp, x, B.jl_empty((ndata, nk), torch.complex128), B.get_fourier_batched(itp, x).clone()))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(20):
        for _, _, out, _ in calls:
            out.fill_(-1)
        torch.cuda.synchronize()
        for which in (0, 1, 0, 1, 2, 0, 2, 1, 0, 1):
            itp, x, out, _ = calls[which]
            with torch.cuda.stream(streams[which % 2]):
                B.get_fourier_batched(itp, x, out=out)
        torch.cuda.synchronize()
        for _, _, out, ref in calls:
            assert torch.equal(out, ref)


@pytest.mark.gpu
def test_uneven_solves():
    """FP64 solves of uneven orders without a read-back, on two streams of one context."""
    import torch

    from epb200 import _lib, synth
    from epb200 import batched as B

    L = _lib.lib()
    ctx = _lib.default_context()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    batches = []
    for seed in (1, 2):
        ns, mats = synth.config3_matrices(400, seed=seed, degenerate_frac=0.25)
        vb = B.VarlenBatch(mats)
        args = (B.ptr(vb.A), B.ptr(vb.a_off), B.ptr(vb.n), len(mats), B.ptr(vb.E), B.ptr(vb.e_off), b"V", 0)
        given = vb.A.clone()
        _lib.check(L.epb_eigh_varlen_async(ctx.h, *args))
        torch.cuda.synchronize()
        batches.append((vb, args, given, vb.A.clone(), vb.E.clone()))
    for _ in range(10):
        for vb, _, given, _, _ in batches:
            vb.A.copy_(given)
            vb.E.fill_(-1)
        torch.cuda.synchronize()
        for s, (_, args, _, _, _) in zip(streams, batches):
            ctx.set_stream(s)
            _lib.check(L.epb_eigh_varlen_async(ctx.h, *args))
        torch.cuda.synchronize()
        for vb, _, _, a, e in batches:
            assert torch.equal(vb.A, a) and torch.equal(vb.E, e)
    assert L.epb_eigh_status(ctx.h) == _lib.EPB_OK
    ctx.set_stream(torch.cuda.current_stream())
