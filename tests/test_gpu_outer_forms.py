"""GPU: real outer axes on both sides of the line between the staged and the
fused form of their FP32 kernels, and short ones in every precision, against
torch's FFT: convolutions, standalone transforms, plain real FFTs."""
import numpy as np
import pytest

from oracle import hybrid as H
from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-13, "ff": 1e-13, "f32": 2e-6}


@pytest.mark.parametrize("precision", ["f64", "ff", "f32"])
@pytest.mark.parametrize("L", [(64, 63, 65), (64, 64, 64), (1, 5, 7),
                               (2, 9, 4), (5, 40, 3), (23, 21, 50),
                               (90, 33, 20)])
def test_real_convolution(native_lib, L, precision):
    import torch
    from fftwpp_gb300.gpu import HybridConvolution
    conv = HybridConvolution([H.REAL, H.PAD, H.PAD], L, precision=precision)
    g = torch.Generator(device="cuda").manual_seed(sum(L))
    f = [torch.randn(L, generator=g, device="cuda", dtype=torch.float64)
         for _ in range(2)]
    got = conv.convolve(*[t.to(conv.dtype) for t in f])[0]
    s = [2 * n for n in L]
    F = [torch.fft.fftn(t, s) for t in f]
    want = torch.fft.ifftn(F[0] * F[1])[:L[0], :L[1], :L[2]].real
    assert rel_l2(got.cpu().numpy().astype(np.float64),
                  want.cpu().numpy()) <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("L,C", [(64, 8190), (64, 8192), (1, 3), (2, 17),
                                 (5, 1), (189, 70)])
def test_real_transforms(native_lib, L, C, precision):
    import torch
    from fftwpp_gb300.gpu import PaddedTransform
    t = PaddedTransform(H.REAL, L, 2 * L, C=C, precision=precision)
    g = torch.Generator(device="cuda").manual_seed(L + C)
    f = torch.randn(L, C, generator=g, device="cuda",
                    dtype=torch.float64)
    F = t.forward(f.to(t.idtype))
    want = torch.fft.rfft(f, t.N, dim=0).conj()
    assert rel_l2(F.cpu().numpy(), want.cpu().numpy()) <= TOL[precision]
    back = t.backward(F).double() / t.N
    assert rel_l2(back.cpu().numpy(), f.cpu().numpy()) <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("n,M", [(256, 4095), (256, 4096), (2, 5), (6, 33),
                                 (420, 7)])
def test_real_ffts(native_lib, n, M, precision):
    import torch
    from fftwpp_gb300 import fft
    g = torch.Generator(device="cuda").manual_seed(n + M)
    rdt = torch.float64 if precision == "f64" else torch.float32
    x = torch.randn(M, n, generator=g, device="cuda", dtype=torch.float64)
    F = fft.mrcfft1d(n, M, precision=precision)
    X = F.fft(x.to(rdt).reshape(F.in_shape))
    want = torch.fft.rfft(x)
    assert rel_l2(X.cpu().numpy().reshape(M, -1),
                  want.cpu().numpy()) <= TOL[precision]
    B = fft.mcrfft1d(n, M, precision=precision)
    y = B.fft(X.reshape(B.in_shape)).double().reshape(M, n) / n
    assert rel_l2(y.cpu().numpy(), x.cpu().numpy()) <= TOL[precision]


@pytest.mark.parametrize("precision", ["f64", "ff", "f32"])
@pytest.mark.parametrize("kinds,L", [
    ([H.CENTERED, H.CENTERED], (170, 511)), ([H.CENTERED, H.CENTERED],
                                             (171, 513)),
    ([H.PAD, H.PAD], (128, 511)), ([H.PAD, H.PAD], (128, 512)),
    ([H.PAD, H.PAD], (128, 513)), ([H.PAD, H.PAD, H.PAD], (9, 21, 48)),
    ([H.PAD, H.PAD], (25, 40)), ([H.CENTERED, H.PAD], (7, 3))])
def test_complex_convolution(native_lib, kinds, L, precision):
    """Complex outer axes around the lines between the forms of their FP32
    (2^18 points a launch) and float-float (2048 columns) kernels."""
    import torch
    from fftwpp_gb300.gpu import HybridConvolution
    conv = HybridConvolution(kinds, L, precision=precision)
    g = torch.Generator(device="cuda").manual_seed(sum(L))
    f = [torch.randn(L, generator=g, device="cuda", dtype=torch.complex128)
         for _ in range(2)]
    got = conv.convolve(*[t.to(conv.dtype) for t in f])[0]
    s = [2 * n for n in L]
    F = [torch.fft.fftn(t, s) for t in f]
    full = torch.fft.ifftn(F[0] * F[1])
    # Centred axes: index i stands for i - L//2, so the product starts at
    # L//2 of the full linear convolution.
    cut = tuple(slice(n // 2, n // 2 + n) if k == H.CENTERED else slice(n)
                for k, n in zip(kinds, L))
    assert rel_l2(got.cpu().numpy().astype(np.complex128),
                  full[cut].cpu().numpy()) <= TOL[precision]
