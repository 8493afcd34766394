"""The tables of the fused transforms (host arithmetic, no GPU), read the way
the kernels read them: the stages in numpy with the library's own twiddle
exponents against numpy's DFT, the positions, the block pairs of real data;
and the padded offsets of Hermitian plans."""
import ctypes

import numpy as np
import pytest

F64, F32, FF = 0, 1, 2


def _tables(lib, n, prec, A=1, herm=0, half=0):
    rad = (ctypes.c_int * 32)()
    k = lib.fgb_fused_radices(n, prec, A, herm, half, rad, 32, None)
    block, inverse = (ctypes.c_long * n)(), (ctypes.c_long * n)()
    pairs, pos, rev = ((ctypes.c_int * m)() for m in (3 * n, n, n))
    nblk = lib.fgb_fused_tables(n, prec, A, herm, half, block, inverse, pairs,
                                pos, rev)
    r = list(rad[:k])
    assert nblk * r[-1] == n
    return (r, np.array(block), np.array(inverse),
            np.array(pairs).reshape(n, 3)[:(nblk + 1) // 2], np.array(pos),
            np.array(rev)[:nblk])


def _dft(R):
    return np.exp(2j * np.pi * np.outer(np.arange(R), np.arange(R)) / R)


CASES = [(n, prec, A, herm, half)
         for n in (1, 2, 7, 12, 36, 48, 60, 105, 160, 210, 256, 384, 768, 1024,
                   1568, 2048)
         for prec, A, herm, half in ((F64, 1, 0, 0), (F64, 2, 1, 0),
                                     (F32, 1, 0, 1), (F32, 4, 1, 0),
                                     (FF, 2, 0, 1), (FF, 5, 1, 0))]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_transform_with_the_tables(native_lib, case):
    n, prec, A, herm, half = case
    radices, block, inverse, _, pos, rev = _tables(native_lib, *case)
    rng = np.random.default_rng(n)
    f = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    W = np.exp(2j * np.pi * np.arange(n) / n)
    R0 = radices[0]
    x, m, nblk = f.copy(), n, 1
    spans = []
    for s, R in enumerate(radices):
        m //= R
        w = np.ones((nblk, R), dtype=complex)
        if s:
            at = nblk - R0 + np.arange((R - 1) * nblk)
            w[:, 1:] = W[block[at]].reshape(R - 1, nblk).T
        x = np.einsum("kr,brm->bkm", _dft(R),
                      x.reshape(nblk, R, m) * w[:, :, None]).ravel()
        spans.append((R, m, nblk))
        nblk *= R
    F = n * np.fft.ifft(f)
    assert np.abs(x[pos] - F).max() <= 1e-13 * n * np.abs(f).max()
    last = radices[-1]
    # Position b R + r holds entry rev(b) + r nblk.
    k = rev[:, None] + np.arange(last)[None, :] * (n // last)
    assert np.array_equal(pos[k.ravel()], np.arange(n))
    z = x.imag + 1j * x.real
    for R, m, nblk in reversed(spans):
        t = np.ones((R, m), dtype=complex)
        at = m - 1 + np.arange((R - 1) * m)
        t[1:] = W[inverse[at]].reshape(R - 1, m)
        z = np.einsum("kr,brm->bkm", _dft(R),
                      z.reshape(nblk, R, m) * t[None]).ravel()
    assert np.abs(z.imag + 1j * z.real - n * f).max() <= \
        1e-13 * n * n * np.abs(f).max()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_block_pairs(native_lib, case):
    """Mode k = kappa + nblk t of a pair's block b has its partner n - k in
    the other block; the first entry holds the blocks that are their own;
    every block is in exactly one place."""
    radices, _, _, pairs, _, rev = _tables(native_lib, *case)
    nblk = len(rev)
    seen = []
    for i, (b, b2, kappa) in enumerate(pairs):
        seen.append(b)
        if i == 0:
            assert b == 0 and kappa == 0 and rev[0] == 0
            assert (b2 < 0) == (nblk % 2 == 1)
            if b2 >= 0:
                assert rev[b2] == nblk // 2
                seen.append(b2)
        else:
            assert rev[b] == kappa and rev[b2] == nblk - kappa
            seen.append(b2)
    assert sorted(seen) == list(range(nblk))


@pytest.mark.parametrize("prec", [F64, F32, FF])
@pytest.mark.parametrize("A", [1, 2, 4, 5])
def test_hermitian_offsets_add_up(native_lib, prec, A):
    """The padded offsets of Hermitian rows' butterflies, for both paddings
    and none, with the partner butterfly of the first stage."""
    for n in list(range(1, 700)) + [768, 1024, 1536, 2048, 4096]:
        rad, lg = (ctypes.c_int * 32)(), (ctypes.c_int * 2)()
        k = native_lib.fgb_fused_radices(n, prec, A, 1, 0, rad, 32, lg)
        if k < 0:
            assert native_lib.fgb_nextfftsize(n) != n
            continue
        for pad in list(lg) + [30]:
            m = n
            for R in rad[:k]:
                m //= R
                i = np.arange(n // R)
                j0 = i + i // m * (R - 1) * m
                step = m + (m >> pad)
                for r in range(R):
                    j = j0 + r * m
                    want = j + (j >> pad)
                    assert np.array_equal(j0 + (j0 >> pad) + r * step, want)
                    assert want.max() < n + ((n - 1) >> pad)
            assert step == 1
