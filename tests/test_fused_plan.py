"""The fused transforms' plans and index arithmetic, restated on the CPU:
radices the kernels hold, padded shared-memory offsets that add up, and the
block-twiddle stages against numpy's DFT."""
import ctypes

import numpy as np
import pytest

F64, F32, FF = 0, 1, 2


def _plan(lib, n, prec, A=1, herm=0, half=0):
    buf = (ctypes.c_int * 32)()
    lg = (ctypes.c_int * 2)()
    k = lib.fgb_fused_radices(n, prec, A, herm, half, buf, 32, lg)
    return None if k < 0 else (list(buf[:k]), list(lg))


def _lengths(lib, top):
    return [n for n in range(1, top) if lib.fgb_nextfftsize(n) == n]


@pytest.mark.parametrize("prec", [F64, F32, FF])
def test_radices_the_kernels_hold(native_lib, prec):
    """Every length has at least two and at most twelve stages; a Hermitian
    first stage is at most 8, and the middle stage's values fit
    its registers."""
    for n in _lengths(native_lib, 5000) + [16384, 19683, 28672]:
        for A in (1, 2, 4, 5, 8):
            for herm, half in ((0, 0), (1, 0), (0, 1)):
                r, _ = _plan(native_lib, n, prec, A, herm, half)
                assert int(np.prod(r)) == n and 2 <= len(r) <= 12
                assert set(r) <= ({1, 2, 3, 4, 5, 6, 7, 8, 16} if prec == F32
                                  else {1, 2, 3, 4, 5, 6, 7, 8})
                assert not herm or r[0] <= 8
                held = r[-1] * (1 if prec == FF else A)
                assert r[-1] in (1, 2, 3, 4) or held <= 20, (n, A, r)
                assert r[-1] != 6
    assert _plan(native_lib, 11, prec) is None


@pytest.mark.parametrize("prec", [F64, F32, FF])
@pytest.mark.parametrize("A", [1, 2, 4, 8])
def test_offsets_add_up(native_lib, prec, A):
    """Input r of a butterfly lies r steps from the padded position of its
    input 0, with the step the kernels compute, for both paddings and none,
    and inside the span they allocate; the last stage's step is 1."""
    for n in _lengths(native_lib, 700) + [768, 1536, 1568, 2048]:
        for half in (0, 1):
            r, pads = _plan(native_lib, n, prec, A, half=half)
            for lg in pads + [30]:
                m = n
                for R in r:
                    m //= R
                    i = np.arange(n // R)
                    j0 = i + i // m * (R - 1) * m
                    step = m + (m >> lg)
                    for k in range(R):
                        j = j0 + k * m
                        want = j + (j >> lg)
                        assert np.array_equal(j0 + (j0 >> lg) + k * step,
                                              want), (n, r, lg)
                        assert want.max() < n + ((n - 1) >> lg)
                assert step == 1


def _rev(radices):
    rev = np.zeros(1, dtype=int)
    mul = 1
    for R in radices:
        rev = (rev[:, None] + mul * np.arange(R)[None, :]).ravel()
        mul *= R
    return rev


@pytest.mark.parametrize("n,prec,half", [(48, F64, 0), (60, F32, 0),
                                         (768, F64, 0), (768, F32, 0),
                                         (1568, F64, 1), (2048, F32, 1),
                                         (105, FF, 0), (7, F64, 0)])
def test_block_twiddle_transform(native_lib, n, prec, half):
    """Forward stages with block twiddles on their inputs leave the sign +1
    spectrum in digit-reversed order; the same butterflies with the inverse
    twiddles, on values with their parts exchanged, take it back."""
    radices, _ = _plan(native_lib, n, prec, half=half)
    rng = np.random.default_rng(n)
    f = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    x, m, nblk = f.copy(), n, 1
    spans = []
    for s, R in enumerate(radices):
        m //= R
        w = np.exp(2j * np.pi * np.outer(_rev(radices[:s]), np.arange(R)) /
                   (nblk * R))
        dft = np.exp(2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)
        v = x.reshape(nblk, R, m) * w[:, :, None]
        x = np.einsum("kr,brm->bkm", dft, v).ravel()
        spans.append((R, m, nblk, dft))
        nblk *= R
    assert np.allclose(x, n * np.fft.ifft(f)[_rev(radices)], rtol=0,
                       atol=1e-10)
    z = x.imag + 1j * x.real
    for R, m, nblk, dft in reversed(spans):
        t = np.exp(2j * np.pi * np.outer(np.arange(R), np.arange(m)) /
                   (R * m))
        z = np.einsum("kr,brm->bkm", dft, z.reshape(nblk, R, m) *
                      t[None]).ravel()
    assert np.allclose(z.imag + 1j * z.real, n * f, rtol=0, atol=1e-9)
