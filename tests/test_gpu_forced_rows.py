"""GPU: few complex rows take a cluster of CTAs each, by a rule on the padded
length and the row count, unless the caller forces m: then the plan runs the
residues it reports."""
import numpy as np
import pytest

from oracle import hybrid as H
from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "ff"])
@pytest.mark.parametrize("kind,L,M,batch,ctas", [
    (H.PAD, 256, 512, 1, 8), (H.PAD, 256, 512, 19, 8),
    (H.PAD, 256, 512, 20, 4), (H.PAD, 512, 1024, 38, 4),
    (H.PAD, 500, 1024, 39, 2), (H.PAD, 500, 1024, 76, 2),
    (H.PAD, 500, 1024, 77, 1), (H.PAD, 200, 400, 1, 1),
    (H.REAL, 512, 1024, 3, 8), (H.CENTERED, 683, 1024, 3, 8)])
def test_ctas_per_row(native_lib, precision, kind, L, M, batch, ctas):
    from fftwpp_gb300.gpu import HybridConvolution
    native_lib.fgb_set_autotune(0)
    try:
        conv = HybridConvolution([kind], [L], [M], batch=batch,
                                 precision=precision)
    finally:
        native_lib.fgb_set_autotune(1)
    if conv.axes[0]["N"] == M:
        assert conv.ctas_per_row == ctas
    assert conv.ctas_per_row in (1, 2, 4, 8)
    f32 = HybridConvolution([kind], [L], [M], batch=batch, precision="f32")
    assert f32.ctas_per_row == 1
    assert ("CTAs/row" in conv.describe()) == (conv.ctas_per_row > 1)


@pytest.mark.parametrize("precision", ["f64", "ff"])
@pytest.mark.parametrize("kind,L,M,m,batch", [
    (H.PAD, 1024, 2048, 512, 1), (H.PAD, 777, 1553, 784, 3),
    (H.CENTERED, 683, 1024, 256, 2), (H.REAL, 600, 1199, 400, 5),
    (H.PAD, 300, 1024, 1024, 1)])
def test_forced_m_runs_as_reported(native_lib, precision, kind, L, M, m,
                                   batch):
    import torch
    from fftwpp_gb300 import gpu
    rng = np.random.default_rng(L + m)
    fs = [rng.uniform(-1, 1, (batch, L)) for _ in range(2)]
    if kind != H.REAL:
        fs = [f + 1j * rng.uniform(-1, 1, f.shape) for f in fs]
    gpu.forget_wisdom()
    for _ in range(2):                     # tuned, then from its record
        conv = gpu.HybridConvolution([kind], [L], [M], m=[m], batch=batch,
                                     precision=precision)
        assert conv.axes[0]["m"] == m and conv.ctas_per_row == 1
        ts = [torch.from_numpy(f.reshape(conv.shape)).cuda() for f in fs]
        got = conv.convolve(*ts)[0].cpu().numpy().reshape(batch, L)
        want = H.convolve([f[-1] for f in fs], [kind], [L], [M])[0]
        assert rel_l2(got[-1], want) <= 1e-13
    # A record of an unforced plan rebuilds it split as it was.
    gpu.forget_wisdom()
    a = gpu.HybridConvolution([kind], [L], [M], batch=batch,
                              precision=precision)
    b = gpu.HybridConvolution([kind], [L], [M], batch=batch,
                              precision=precision)
    assert a.ctas_per_row == b.ctas_per_row
    gpu.forget_wisdom()
