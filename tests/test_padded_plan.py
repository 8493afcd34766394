"""Column tiles of standalone padded transforms (host planning, no GPU): the
two-buffer kernels they launch fit a CTA's shared memory at the planned tile,
both ways, whatever the fold and residue counts."""
import ctypes

import pytest

SMEM_MAX = 227 * 1024
F64, F32 = 0, 1
PAD, CENTERED = 0, 1


def _padded(n):
    return n + n // 32 + 1


def _tiles(lib, kind, L, M, C, m, prec):
    h = lib.fgb_pad_create(kind, L, M, C, m, prec)
    if not h:
        return None
    info = (ctypes.c_long * 10)()
    assert lib.fgb_pad_info(h, info) == 0
    lib.fgb_pad_destroy(h)
    return list(info)


def _needs(v, prec):
    """Bytes of the forward and backward kernels: two padded transform
    buffers, the second holding the input block, and an accumulator where
    there are several residues."""
    m, _, q, _, L, _, _, _, tile, tileB = v
    e = 16 if prec == F64 else 8
    fwd = _padded(m * tile) + max(_padded(m * tile), L * tile)
    bwd = 2 * _padded(m * tileB) + (L * tileB if q > 1 else 0)
    return e * fwd, e * bwd


@pytest.mark.parametrize("prec", [F64, F32])
@pytest.mark.parametrize("C", [1, 5, 4096])
@pytest.mark.parametrize("kind", [PAD, CENTERED])
def test_padded_tiles_fit(native_lib, kind, C, prec):
    planned = 0
    for L in list(range(500, 5200, 50)) + [600, 2400, 2500]:
        M = 2 * L - 1 if kind == PAD else 3 * ((L + 1) // 2) - 2 * (L % 2)
        for m in (0, native_lib.fgb_nextfftsize(M),
                  native_lib.fgb_nextfftsize(L)):
            v = _tiles(native_lib, kind, L, M, C, m, prec)
            if v is None:
                assert m > 0                   # a forced m may be too long
                continue
            assert max(_needs(v, prec)) <= SMEM_MAX, (L, m, v)
            planned += 1
    assert planned >= 90


@pytest.mark.parametrize("prec", [F64, F32])
def test_real_axis_too_long_is_refused_at_creation(native_lib, prec):
    """The longest real axis is where two padded buffers of one column fill
    shared memory; the next length is no plan, rather than one that fails
    every run."""
    from fftwpp_gb300 import _native
    e = 16 if prec == F64 else 8
    REAL = 3
    took = refused = 0
    for L in range(5000, 20000, 250):
        M = 2 * L - 1
        N = M + 1
        while native_lib.fgb_nextfftsize(N // 2) != N // 2:
            N += 2
        v = _tiles(native_lib, REAL, L, M, 1, 0, prec)
        if 2 * e * _padded(N // 2 + 1) <= SMEM_MAX:
            assert v and v[3] == N, L
            took += 1
        else:
            assert v is None and "too long" in _native.last_error()
            refused += 1
    assert took >= 8 and refused >= 8
