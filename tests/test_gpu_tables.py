"""GPU: twiddle tables are made with their plan.  A table that cannot be
allocated is an error of the creation, and a created plan's first run
allocates nothing, so that it may be the one that a CUDA graph captures.
Tables stay cached for the process: lengths that few tests share."""
import numpy as np
import pytest

from oracle import hybrid as H
from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu


def _conv(kinds, L, **kw):
    from fftwpp_gb300.gpu import HybridConvolution
    if kinds[-1] == H.HERMITIAN:
        kw.setdefault("mult", "realbinary")
    return lambda: HybridConvolution(kinds, L, **kw)


def _padded(kind, L, **kw):
    def make():
        from fftwpp_gb300.gpu import PaddedTransform
        return PaddedTransform(kind, L, **kw)
    return make


def _plain(name, *args):
    def make():
        from fftwpp_gb300 import fft
        return getattr(fft, name)(*args)
    return make


PLANS = {
    "direct-row": _conv([H.PAD], [2917], batch=300),
    "split-row": _conv([H.PAD], [2593]),
    "residues": _conv([H.PAD], [2713], m=[1225], batch=300),
    "long-row": _conv([H.PAD], [60011], precision="f32"),
    "hermitian": _conv([H.CENTERED, H.HERMITIAN], [173, 691]),
    "folded-outer": _conv([H.PAD, H.PAD], [1471, 29], m=[245, 0]),
    "real-outer": _conv([H.REAL, H.PAD, H.PAD], [37, 53, 61],
                        precision="ff"),
    "padded": _padded(H.CENTERED, 2269, C=3),
    "padded-real": _padded(H.REAL, 1951, C=3),
    "fft": _plain("fft1d", 6174, -1),
    "fft-two-pass": _plain("fft1d", 38416, 1),
    "rcfft": _plain("rcfft1d", 4802),
}


def _call(plan):
    """(run(out), inputs, out) of a plan on random inputs."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(1)

    def rand(shape, dtype):
        return torch.randn(shape, generator=gen, device="cuda", dtype=dtype)
    name = type(plan).__name__
    if name == "HybridConvolution":
        ins = [rand(plan.shape, plan.dtype) for _ in range(plan.A)]
        return (lambda o: plan.convolve(*ins, out=[o]), ins,
                torch.zeros_like(ins[0]))
    if name == "PaddedTransform":
        f = rand((plan.stored, plan.C), plan.idtype)
        return (lambda o: plan.forward(f, out=o), [f],
                torch.zeros((plan.rows, plan.C), dtype=plan.cdtype,
                            device="cuda"))
    x = rand(plan.in_shape, plan.in_dtype)
    return (lambda o: plan.fft(x, out=o), [x],
            torch.zeros(plan.out_shape, dtype=plan.out_dtype, device="cuda"))


def _want(label, plan, ins):
    """The result in plain torch, where that is one line."""
    import torch
    name = type(plan).__name__
    if name == "HybridConvolution":
        if H.HERMITIAN in plan.kinds:
            return None
        first = plan.shape[1:] if plan.batch > 1 else plan.shape
        dims = list(range(-len(first), 0))
        F = [torch.fft.fftn(t, [2 * n for n in first], dims) for t in ins]
        h = torch.fft.ifftn(F[0] * F[1], dim=dims)
        h = h[(Ellipsis,) + tuple(slice(n) for n in first)]
        return h if ins[0].is_complex() else h.real
    if name != "PaddedTransform":
        x = ins[0]
        if plan.in_dtype != plan.out_dtype:
            return torch.fft.rfft(x)
        return torch.fft.fft(x) if label == "fft" else \
            torch.fft.ifft(x) * x.numel()
    return None


@pytest.mark.parametrize("name", list(PLANS))
def test_tables_are_made_with_the_plan(native_lib, name):
    import torch
    make = PLANS[name]
    native_lib.fgb_set_autotune(0)
    try:
        plan, k = None, 0
        while plan is None:
            native_lib.fgb_debug_fail_allocation_after(k)
            try:
                plan = make()
            except ValueError as e:
                assert "allocation" in str(e) or "memory" in str(e), str(e)
                k += 1
                assert k < 40
            finally:
                native_lib.fgb_debug_fail_allocation_after(-1)
    finally:
        native_lib.fgb_set_autotune(1)
    run, ins, out = _call(plan)
    torch.cuda.synchronize()
    native_lib.fgb_debug_fail_allocation_after(0)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            run(out)
    finally:
        native_lib.fgb_debug_fail_allocation_after(-1)
    graph.replay()
    got = out.clone()
    out.zero_()
    run(out)
    assert torch.equal(got, out) and bool(got.abs().max() > 0)
    want = _want(name, plan, ins)
    if want is not None:
        tol = 2e-6 if got.dtype in (torch.complex64, torch.float32) else 1e-13
        assert rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= tol


def test_batch_tables_are_made_with_the_plan(native_lib):
    import torch
    from fftwpp_gb300.gpu import BatchedConvolution
    lengths = [1777, 70001, 61]
    conv, k = None, 0
    while conv is None:
        native_lib.fgb_debug_fail_allocation_after(k)
        try:
            conv = BatchedConvolution(lengths)
        except ValueError as e:
            assert "allocation" in str(e) or "memory" in str(e), str(e)
            k += 1
            assert k < 60
        finally:
            native_lib.fgb_debug_fail_allocation_after(-1)
    rng = np.random.default_rng(3)
    f, g = (rng.uniform(-1, 1, sum(lengths)) +
            1j * rng.uniform(-1, 1, sum(lengths)) for _ in range(2))
    got = conv.convolve(torch.from_numpy(f).cuda(),
                        torch.from_numpy(g).cuda())[0].cpu().numpy()
    at = 0
    for n in lengths:
        a, b = f[at:at + n], g[at:at + n]
        want = np.fft.ifft(np.fft.fft(a, 2 * n) * np.fft.fft(b, 2 * n))[:n]
        assert rel_l2(got[at:at + n], want) <= 1e-13
        at += n
