"""Few complex rows, each split over a cluster of CTAs: every cluster size and
the plans next to the rule's lines against the CPU oracle, in place too."""
import numpy as np
import pytest

from oracle import hybrid as H
from oracle.direct import rel_l2

pytestmark = pytest.mark.gpu

# (kind, L, M, batch, mult, A): eight, four and two CTAs a row, one; padded
# lengths at the line (512), odd multiples of the cluster, several residues.
CASES = [(H.PAD, 256, None, 1, "binary", 2),
         (H.PAD, 255, 511, 19, "binary", 2),
         (H.PAD, 1024, None, 20, "binary", 2),
         (H.PAD, 777, None, 38, "correlation", 2),
         (H.PAD, 500, None, 76, "binary", 2),
         (H.PAD, 500, None, 77, "binary", 2),
         (H.CENTERED, 683, None, 3, "binary", 2),
         (H.CENTERED, 3000, None, 2, "binary", 2),
         (H.PAD, 3000, None, 1, "binary", 2),
         (H.REAL, 600, None, 5, "binary", 2),
         (H.PAD, 300, None, 2, "dot", 4)]


@pytest.mark.parametrize("precision", ["f64", "ff"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_split_rows(native_lib, case, precision):
    import torch
    from fftwpp_gb300.gpu import HybridConvolution
    kind, L, M, batch, mult, A = case
    conv = HybridConvolution([kind], [L], None if M is None else [M],
                             A=A, mult=mult, precision=precision, batch=batch)
    rng = np.random.default_rng(L + batch)
    fs = [rng.uniform(-1, 1, (batch, L)) for _ in range(A)]
    if kind != H.REAL:
        fs = [f + 1j * rng.uniform(-1, 1, f.shape) for f in fs]
    ts = [torch.from_numpy(f.reshape(conv.shape)).cuda() for f in fs]
    conv.convolve(*ts, out=[ts[0]])             # over the first input
    got = ts[0].cpu().numpy().reshape(batch, L)
    rows = range(batch) if L < 400 else sorted({0, batch // 2, batch - 1})
    for k in rows:
        want = H.convolve([f[k] for f in fs], [kind], [L], conv.M,
                          mult=mult)[0]
        assert rel_l2(got[k], want) <= 1e-13, k
