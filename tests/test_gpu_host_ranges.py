"""GPU: a float-float host call whose outer transforms run in column ranges
takes the same form of its kernels as the device call over all columns, below
and above the line between the two forms, and gives the same bits."""
import numpy as np
import pytest

from oracle import hybrid as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds,L", [([H.PAD, H.PAD], [24, 1500]),
                                     ([H.PAD, H.CENTERED], [40, 2051]),
                                     ([H.PAD, H.PAD], [24, 700]),
                                     ([H.PAD, H.PAD, H.PAD], [20, 30, 70])])
@pytest.mark.parametrize("guard", [1, 0])
def test_ranges_equal_device_call(native_lib, kinds, L, guard):
    import torch
    from fftwpp_gb300.gpu import HybridConvolution
    rng = np.random.default_rng(L[-1])
    fs = [rng.uniform(-1, 1, L) + 1j * rng.uniform(-1, 1, L)
          for _ in range(2)]
    native_lib.fgb_set_ff_range_guard(guard)
    try:
        conv = HybridConvolution(kinds, L, precision="ff")
        want = conv.convolve(*[torch.from_numpy(f).cuda() for f in fs])[0]
        want = want.cpu().numpy()
        for wi in (0, 1, 2):
            for wo in (0, 1, 2):
                native_lib.fgb_set_host_path(wi, wo)
                h = [torch.from_numpy(f.copy()).pin_memory().numpy()
                     for f in fs]
                conv.convolve_host(*h)
                assert np.array_equal(h[0], want), (wi, wo)
    finally:
        native_lib.fgb_set_host_path(-1, -1)
        native_lib.fgb_set_ff_range_guard(1)
