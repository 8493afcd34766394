"""GPU: Hermitian rows through every form of their kernels (ping-pong, staged,
fused: by precision, inputs and length) against numpy's real FFT, in place,
with row counts that leave a group part full."""
import numpy as np
import pytest

from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-13, "ff": 1e-13, "f32": 2e-6}


def _product(u, mult):
    if mult == "realbinary":
        return [u[0] * u[1]]
    if mult == "realjacobian":
        return [u[0] * u[3] - u[1] * u[2]]
    return [u[4] * u[3], -u[4] * u[2], -u[4] * u[1], u[4] * u[0]]


@pytest.mark.parametrize("precision", ["f64", "f32", "ff"])
@pytest.mark.parametrize("A,B,mult", [(2, 1, "realbinary"),
                                      (4, 1, "realjacobian"),
                                      (5, 4, "realjacadj")])
@pytest.mark.parametrize("H,rows", [(1, 1), (2, 5), (9, 50), (25, 7),
                                    (90, 301), (160, 33), (250, 9), (256, 5),
                                    (300, 3), (384, 2)])
def test_hermitian_rows(native_lib, H, rows, A, B, mult, precision):
    import torch
    from fftwpp_gb300.gpu import HERMITIAN, HybridConvolution
    conv = HybridConvolution([HERMITIAN], [2 * H - 1], [3 * H - 2], A=A, B=B,
                             mult=mult, precision=precision, batch=rows)
    rng = np.random.default_rng(H + rows)
    f = [rng.uniform(-1, 1, (rows, H)) + 1j * rng.uniform(-1, 1, (rows, H))
         for _ in range(A)]
    for a in f:
        a[:, 0] = a[:, 0].real
    t = [torch.from_numpy(a).reshape(conv.shape).to(conv.dtype).cuda()
         for a in f]
    conv.convolve(*t, out=t[:B])
    N = 3 * H + 3 + (3 * H + 3) % 2
    u = [np.fft.irfft(np.concatenate([a, np.zeros((rows, N // 2 + 1 - H))], 1),
                      N) * N for a in f]
    for got, w in zip(t, _product(u, mult)):
        want = np.fft.rfft(w)[:, :H] / N
        assert rel_l2(got.cpu().numpy().reshape(rows, H)
                      .astype(np.complex128), want) <= TOL[precision]
