"""Padded length of a convolution's innermost axis (host planning, no GPU):
where the outputs depend on it (M below the dealiasing length, a caller's
functor) it is the one that the staged rows' estimate picks, restated here;
above, any length holds the same convolution."""
import ctypes

import numpy as np
import pytest

PAD, CENTERED, HERMITIAN, REAL = range(4)
F64, F32, FF = 0, 1, 2
BINARY, REALBINARY, CORRELATION, USER = 1, 2, 3, 9
SMEM_MAX = 227 * 1024


def _row(lib, kind, L, M, A=2, B=1, mult=BINARY, prec=F64, m=0):
    v = (ctypes.c_long * 4)()
    rc = lib.fgb_row_length(kind, L, M, m, A, B, mult, prec, v)
    assert rc >= 0
    return list(v) if rc else None


def _instr(n):
    """Instructions of a staged transform: codelet and twiddles per point."""
    rad = []
    for f in (8, 8, 8, 8, 8, 4, 2) + (7,) * 5 + (5,) * 5 + (3,) * 8:
        if n % f == 0:
            rad.append(f)
            n //= f
    assert n == 1
    code = {8: 7, 4: 4, 2: 2, 3: 4.7, 5: 6.8, 7: 8.6}
    return int(np.prod(rad)) * sum(code[R] + (4 * (R - 1) / R if i else 0)
                                   for i, R in enumerate(rad))


def _staged(lib, L, M, A, B, prec):
    """Length of the cheapest staged plan that fits shared memory."""
    best = None
    e, nbuf = (8, 1) if prec == F32 else (16, 2 if prec == F64 else 1)
    for q in range(1, 65):
        m = lib.fgb_nextfftsize(-(-M // q))
        n = m * A
        if e * ((A + B) * L + nbuf * (n + n // 32 + 1)) > SMEM_MAX:
            continue
        p = -(-L // m)
        c = (q * (A + B) * _instr(m) + A * m * (2 * p + (q - 1) * 6 * p) +
             B * L * (2 + (q - 1) * 6))
        if best is None or c < best[0] * (1 - 1e-12):
            best = (c, m * q)
    return best and best[1]


@pytest.mark.parametrize("prec", [F64, F32, FF])
@pytest.mark.parametrize("kind,A,B,mult", [(PAD, 2, 1, BINARY),
                                           (CENTERED, 2, 1, CORRELATION),
                                           (PAD, 4, 2, USER),
                                           (PAD, 2, 1, REALBINARY)])
def test_length_stays_where_outputs_depend_on_it(native_lib, kind, A, B, mult,
                                                 prec):
    seen = 0
    for M in list(range(1, 400)) + [441, 625, 1023, 1024, 2401, 3001]:
        for L in sorted({M, max(1, 3 * M // 4)}):
            v = _row(native_lib, kind, L, M, A, B, mult, prec)
            want = _staged(native_lib, L, M, A, B, prec)
            if v is None:
                assert want is None
                continue
            if v[3]:
                assert v[2] >= M and mult != USER and mult != REALBINARY
                continue
            assert v[2] == want and v[0] * v[1] == v[2], (L, M, v)
            seen += 1
    assert seen >= 390


@pytest.mark.parametrize("prec", [F64, F32, FF])
def test_hermitian_length_stays(native_lib, prec):
    """The least even length with a smooth half below 3H-2, and where the
    multiplier is not one for real grid values."""
    def least(M):
        N = max(2, M + M % 2)
        while native_lib.fgb_nextfftsize(N // 2) != N // 2:
            N += 2
        return N
    for L in range(1, 300):
        H = (L + 1) // 2
        for M, mult in ((L, REALBINARY), (3 * H - 3, REALBINARY),
                        (3 * H - 2, BINARY), (3 * H - 2, USER)):
            if M < L:
                continue
            v = _row(native_lib, HERMITIAN, L, M, mult=mult, prec=prec)
            if not v[3]:
                assert v[2] == least(M), (L, M, mult)
            else:
                assert mult == REALBINARY and M >= 3 * H - 2


@pytest.mark.parametrize("kind", [PAD, CENTERED, HERMITIAN])
@pytest.mark.parametrize("correlate", [0, 1])
def test_any_length_line(native_lib, kind, correlate):
    """On the line the products of all stored modes leave no alias in the
    stored range, and one below it they do."""
    for L in range(2, 40):
        H = (L + 1) // 2
        lo = {PAD: 0, CENTERED: -(L // 2), HERMITIAN: 1 - H}[kind]
        hi = H - 1 if kind == HERMITIAN else lo + L - 1
        mult = REALBINARY if kind == HERMITIAN else \
            CORRELATION if correlate else BINARY
        free = [M for M in range(L, 3 * L + 2)
                if _row(native_lib, kind, L, M, mult=mult)[3]]
        assert free == list(range(free[0], 3 * L + 2))

        def aliases(N):
            a = np.arange(lo, hi + 1)
            s = np.unique(a[:, None] - a[None, :] if correlate else
                          a[:, None] + a[None, :])
            return any(lo <= k + w * N <= hi for k in s for w in (-2, -1, 1, 2))
        assert not any(aliases(N) for N in range(free[0], free[0] + L))
        if free[0] > L and not (correlate and kind == HERMITIAN):
            assert aliases(free[0] - 1), (kind, L, free[0])
