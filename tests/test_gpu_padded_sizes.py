"""GPU: standalone padded transforms whose data fill one residue block of 900
to 5000 points, where the two-buffer kernels need a narrower tile than the
one-buffer ones: backward(forward(f)) = N f."""
import numpy as np
import pytest

from oracle import hybrid as H

pytestmark = pytest.mark.gpu

CASES = [(H.PAD, 2500, 1, 0), (H.CENTERED, 2400, 1, 0),
         (H.CENTERED, 600, 4096, 0), (H.PAD, 600, 4096, 0),
         (H.PAD, 600, 4096, 1200), (H.CENTERED, 3300, 1, 5000),
         (H.PAD, 4900, 3, 0), (H.CENTERED, 1201, 517, 0)]


@pytest.mark.parametrize("precision,tol", [("f64", 1e-13), ("f32", 2e-6)])
@pytest.mark.parametrize("kind,L,C,m", CASES)
def test_roundtrip_one_block(native_lib, kind, L, C, m, precision, tol):
    import torch
    from fftwpp_gb300.gpu import PaddedTransform
    t = PaddedTransform(kind, L, C=C, m=m, precision=precision)
    rng = np.random.default_rng(L + C)
    f = torch.from_numpy(rng.uniform(-1, 1, (L, C)) +
                         1j * rng.uniform(-1, 1, (L, C))).to(t.idtype).cuda()
    g = t.backward(t.forward(f))
    err = float(torch.linalg.norm(g / t.N - f) / torch.linalg.norm(f))
    assert err <= tol
