"""GPU: convolutions padded below the dealiasing length, whose outputs alias:
the same padded length with and without timing, from a wisdom record of
another length, and for a functor's plan, and the cyclic convolution of that
length in numpy."""
import numpy as np
import pytest

from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu


def _conv(L, M, precision="f64", mult="binary", batch=1):
    from fftwpp_gb300.gpu import PAD, HybridConvolution
    return HybridConvolution([PAD], [L], [M], mult=mult, precision=precision,
                             batch=batch)


@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), ("f32", 2e-6),
                                           ("ff", 1e-13)])
@pytest.mark.parametrize("L,M", [(21, 21), (49, 49), (40, 49), (343, 343),
                                 (735, 735), (300, 441), (25, 31)])
def test_aliased_rows(native_lib, L, M, precision, tol):
    import torch
    from fftwpp_gb300 import gpu
    rng = np.random.default_rng(L)
    f, g = (rng.uniform(-1, 1, L) + 1j * rng.uniform(-1, 1, L)
            for _ in range(2))
    lengths = set()
    try:
        for tuned in (False, True):
            gpu.forget_wisdom()
            native_lib.fgb_set_autotune(int(tuned))
            for batch in (1, 200):
                conv = _conv(L, M, precision, batch=batch)
                N = conv.axes[0]["N"]
                lengths.add(N)
                t = [torch.from_numpy(np.tile(a, (batch, 1))
                                      .reshape(conv.shape))
                     .to(conv.dtype).cuda() for a in (f, g)]
                got = conv.convolve(*t)[0].cpu().numpy().reshape(batch, L)
                want = np.fft.ifft(np.fft.fft(f, N) * np.fft.fft(g, N))[:L]
                assert rel_l2(got[-1].astype(np.complex128), want) <= tol
        lengths.add(_conv(L, M, precision, mult="user").axes[0]["N"])
    finally:
        native_lib.fgb_set_autotune(1)
        gpu.forget_wisdom()
    assert len(lengths) == 1


def test_wisdom_of_another_length(native_lib):
    """A record whose m makes another padded length is not taken where the
    outputs depend on it, and is where they do not."""
    from fftwpp_gb300 import gpu
    try:
        for M, m in ((49, 64), (97, 128)):
            gpu.forget_wisdom()
            N = _conv(49, M).axes[0]["N"]
            key, value = gpu.export_wisdom().rstrip("\n").split("\t")
            v = value.split()
            v[0] = str(m)
            gpu.forget_wisdom()
            gpu.import_wisdom(f"{key}\t{' '.join(v)}\n")
            got = _conv(49, M).axes[0]
            assert got["N"] == (N if M == 49 else m)
    finally:
        gpu.forget_wisdom()
