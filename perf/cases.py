"""The convolutions this library is used for, as cases that can be timed and
checked: sizes, precisions and entry points of its benchmark and tests, from
one small problem to the 3D one.

A case names its family and sizes:
  conv    gpu.HybridConvolution on device tensors (1D batches, 2D, 3D)
  host    the same plan called on page-locked host arrays (the C entry)
  uneven  gpu.BatchedConvolution, many 1D problems of uneven lengths
  grad    autograd.GraphedLossStep, Jacobian forward and adjoint
"""
import ctypes
import math

import numpy as np
import torch

from fftwpp_gb300 import _native
from fftwpp_gb300.autograd import AdvectionJacobian, GraphedLossStep
from fftwpp_gb300.gpu import (CENTERED, HERMITIAN, PAD, REAL,
                              BatchedConvolution, HybridConvolution)

KINDS = {"pad": PAD, "centered": CENTERED, "hermitian": HERMITIAN,
         "real": REAL}


def listed():
    return [
        # One small convolution at a time, as a caller in a loop makes it:
        # the launch and the latency of one CTA are all there is.
        dict(name="conv1d_one_f64", family="conv", kinds="pad", L="1024",
             batch=1, precision="f64"),
        # Thousands of equal pairs at once: filter banks, spectral products.
        dict(name="conv1d_4096_f32", family="conv", kinds="pad", L="1024",
             batch=4096, precision="f32"),
        # The same in the drop-in precision with lengths nobody rounded.
        dict(name="conv1d_ragged_f64", family="conv", kinds="pad", L="777",
             batch=300, precision="f64"),
        # The nonlinear term of a 2D pseudospectral solver, in the drop-in
        # precision and in the two faster ones.
        dict(name="hconv2d_1023_f64", family="conv",
             kinds="centered hermitian", L="1023 1023", batch=1,
             precision="f64"),
        dict(name="hconv2d_1023_f32", family="conv",
             kinds="centered hermitian", L="1023 1023", batch=1,
             precision="f32"),
        dict(name="hconv2d_1023_ff", family="conv",
             kinds="centered hermitian", L="1023 1023", batch=1,
             precision="ff"),
        # Complex images of odd sizes.
        dict(name="conv2d_ragged_f64", family="conv", kinds="pad pad",
             L="413 389", batch=1, precision="f64"),
        # Real volumes: the largest workload, and one of uneven sides in the
        # drop-in precision.
        dict(name="real3d_256_f32", family="conv", kinds="real pad pad",
             L="256 256 256", batch=1, precision="f32"),
        dict(name="real3d_ragged_f64", family="conv", kinds="real pad pad",
             L="127 90 101", batch=1, precision="f64"),
        # 512 signals of lengths from tens to tens of thousands, one launch.
        dict(name="uneven_512_f32", family="uneven", count=512, lo=64,
             hi=65536, lengths=2024, precision="f32"),
        # A C program's call on its own (page-locked) arrays, modest size.
        dict(name="hconv2d_host_255_f64", family="host",
             kinds="centered hermitian", L="255 255", batch=1,
             precision="f64"),
        # A training step: advection Jacobian, loss and both gradients.
        dict(name="grad_1023_f32", family="grad", Lx=1023, Ly=1023,
             precision="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(n):
    return n | 1


def draw(rng):
    family = rng.choice(["conv1d", "conv1d", "conv2d", "hconv2d", "hconv2d",
                         "conv3d", "uneven", "host", "grad"])
    if family == "conv1d":
        return dict(family="conv", kinds=rng.choice(["pad", "centered"]),
                    L=str(_log(rng, 48, 3000)), batch=_log(rng, 1, 2500),
                    precision=rng.choice(["f64", "f32", "ff"]))
    if family == "conv2d":
        return dict(family="conv",
                    kinds=rng.choice(["pad pad", "centered centered"]),
                    L="%d %d" % (_log(rng, 24, 900), _log(rng, 24, 900)),
                    batch=1, precision=rng.choice(["f64", "f32", "ff"]))
    if family == "hconv2d":
        return dict(family="conv", kinds="centered hermitian",
                    L="%d %d" % (_odd(_log(rng, 31, 1200)),
                                 _odd(_log(rng, 31, 1200))),
                    batch=1, precision=rng.choice(["f64", "f32", "ff"]))
    if family == "conv3d":
        return dict(family="conv", kinds="real pad pad",
                    L="%d %d %d" % tuple(_log(rng, 20, 200)
                                         for _ in range(3)),
                    batch=1, precision=rng.choice(["f64", "f32", "ff"]))
    if family == "uneven":
        return dict(family="uneven", count=_log(rng, 24, 400), lo=64,
                    hi=_log(rng, 1000, 65536), lengths=rng.randrange(1 << 20),
                    precision=rng.choice(["f64", "f32"]))
    if family == "host":
        return dict(family="host", kinds="centered hermitian",
                    L="%d %d" % (_odd(_log(rng, 31, 800)),
                                 _odd(_log(rng, 31, 800))),
                    batch=1, precision=rng.choice(["f64", "ff"]))
    return dict(family="grad", Lx=_odd(_log(rng, 63, 1100)),
                Ly=_odd(_log(rng, 63, 1100)),
                precision=rng.choice(["f64", "f32", "ff"]))


# ---------------------------------------------------------------------------
# Sizes and inputs.

def _axes(case):
    return ([KINDS[k] for k in case["kinds"].split()],
            [int(n) for n in case["L"].split()])


def _stored(kind, n):
    return (n + 1) // 2 if kind == HERMITIAN else n


def _padded(kind, n):
    """The minimum padded length: the 3/2 rule for centred data, else the
    full linear convolution."""
    if kind in (CENTERED, HERMITIAN):
        return 3 * ((n + 1) // 2) - 2 * (n % 2)
    return 2 * n - 1


def _lengths(case):
    r = np.random.default_rng(case["lengths"])
    return [int(round(math.exp(u))) for u in
            r.uniform(math.log(case["lo"]), math.log(case["hi"]),
                      case["count"])]


def _complex(case):
    return torch.complex64 if case["precision"] == "f32" else torch.complex128


def _real(case):
    return torch.float32 if case["precision"] == "f32" else torch.float64


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(shape, case, g):
    """iid complex U[-1,1]."""
    x = torch.rand(*shape, 2, generator=g, device="cuda", dtype=torch.float64)
    return torch.view_as_complex(2 * x - 1).to(_complex(case)).contiguous()


def _symmetrize(f):
    """Hermitian symmetry of the k_y = 0 column of centred modes (odd Lx)."""
    x0 = f.shape[0] // 2
    col = f[:, 0].clone()
    f[:x0, 0] = col[x0 + 1:].flip(0).conj()
    f[x0, 0] = col[x0].real
    return f


def _fields(case, seed):
    kinds, L = _axes(case)
    shape = [_stored(k, n) for k, n in zip(kinds, L)]
    if case["batch"] > 1:
        shape = [case["batch"]] + shape
    g = _generator(seed)
    if kinds[0] == REAL:
        return [torch.randn(*shape, generator=g, device="cuda",
                            dtype=torch.float64).to(_real(case))
                for _ in range(2)]
    fs = [_uniform(shape, case, g) for _ in range(2)]
    if kinds[-1] == HERMITIAN:
        fs = [_symmetrize(f) for f in fs]
    return fs


def _spectra(case, seed):
    """psi and omega with amplitudes |k|^-2 and random phases."""
    Lx, Ly = case["Lx"], case["Ly"]
    H = (Ly + 1) // 2
    kx = (torch.arange(Lx, device="cuda", dtype=torch.float64) -
          Lx // 2)[:, None]
    ky = torch.arange(H, device="cuda", dtype=torch.float64)[None, :]
    k2 = kx * kx + ky * ky
    amp = torch.where(k2 > 0, 1 / torch.clamp(k2, min=1), torch.zeros_like(k2))
    g = _generator(seed)
    out = []
    for _ in range(2):
        ph = 2 * math.pi * torch.rand(Lx, H, generator=g, device="cuda",
                                      dtype=torch.float64)
        out.append(_symmetrize(torch.polar(amp, ph)).to(_complex(case)))
    return out


# ---------------------------------------------------------------------------

def prepare(case, seed):
    family = case["family"]
    if family == "uneven":
        Ls = _lengths(case)
        plan = BatchedConvolution(Ls, precision=case["precision"], tune=True)
        g = _generator(seed)
        fs = [_uniform([sum(Ls)], case, g) for _ in range(2)]
        return dict(family=family, plan=plan, inputs=fs)
    if family == "grad":
        op = AdvectionJacobian(case["Lx"], case["Ly"], case["precision"])
        step = GraphedLossStep(op, *_spectra(case, seed))
        return dict(family=family, op=op, step=step)
    kinds, L = _axes(case)
    plan = HybridConvolution(
        kinds, L, mult="realbinary" if kinds[-1] == HERMITIAN else "binary",
        precision=case["precision"], batch=case["batch"])
    fs = _fields(case, seed)
    if family == "host":
        host = []
        for f in fs:
            h = torch.empty(f.shape, dtype=f.dtype, pin_memory=True)
            h.copy_(f)
            host.append(h)
        out = torch.empty(fs[0].shape, dtype=fs[0].dtype, pin_memory=True)
        ins = (ctypes.c_void_p * 2)(*[h.data_ptr() for h in host])
        outs = (ctypes.c_void_p * 1)(out.data_ptr())
        return dict(family=family, plan=plan, host=host, out=out, ins=ins,
                    outs=outs)
    return dict(family=family, plan=plan, inputs=fs)


def run(state):
    family = state["family"]
    if family == "grad":
        loss, gp, go = state["step"]()
        return [loss, gp, go]
    if family == "host":
        rc = state["plan"].lib.fgb_convolve_host(state["plan"].handle,
                                                 state["ins"], state["outs"])
        if rc != 0:
            raise RuntimeError(_native.last_error())
        return [state["out"]]
    return state["plan"].convolve(*state["inputs"])


def _fft_flops(n):
    return 5.0 * n * math.log2(max(n, 2))


def work(case):
    """Each input read and each output written once; the padded transforms
    of every input and output, over the rows that hold data."""
    elem = 8 if case["precision"] == "f32" else 16
    if case["family"] == "uneven":
        Ls = _lengths(case)
        return {"bytes": 3 * elem * sum(Ls),
                "flops": sum(3 * _fft_flops(2 * n - 1) for n in Ls)}
    if case["family"] == "grad":
        kinds, L, batch = [CENTERED, HERMITIAN], [case["Lx"], case["Ly"]], 1
        transforms = (4 + 1) + (5 + 4)
        arrays = 2 + 2                       # psi, omega and their gradients
    else:
        kinds, L = _axes(case)
        batch, transforms, arrays = case["batch"], 3, 3
    n = [_stored(k, l) for k, l in zip(kinds, L)]
    N = [_padded(k, l) for k, l in zip(kinds, L)]
    if kinds[0] == REAL:
        elem //= 2
    half = [0.5 if k in (HERMITIAN, REAL) else 1.0 for k in kinds]
    flops, rows = 0.0, float(batch)          # rows: transformed outer lines
    for d in range(len(n)):
        lines = rows
        for e in range(d + 1, len(n)):
            lines *= n[e]
        flops += lines * half[d] * _fft_flops(N[d])
        rows *= N[d] // 2 + 1 if kinds[d] == REAL else N[d]
    size = batch
    for v in n:
        size *= v
    return {"bytes": arrays * elem * size, "flops": transforms * flops}


# ---------------------------------------------------------------------------
# The same results from zero-padded transforms in 64 bits.

def _smooth(n):
    while True:
        r = n
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            return n
        n += 1


def _hermitian_grid(f, Nx, Ny):
    """Physical values sum_k f_k e^{ik.x} of centred Hermitian modes."""
    Lx, H = f.shape
    idx = (torch.arange(Lx, device=f.device) - Lx // 2) % Nx
    z = torch.zeros(Nx, Ny // 2 + 1, dtype=torch.complex128, device=f.device)
    z = z.index_put((idx[:, None], torch.arange(H, device=f.device)[None, :]),
                    f)
    return torch.fft.irfft(torch.fft.ifft(z, dim=0), n=Ny, dim=1) * (Nx * Ny)


def _hermitian_modes(u, Lx, H):
    Nx, Ny = u.shape
    z = torch.fft.fft(torch.fft.rfft(u, dim=1), dim=0) / (Nx * Ny)
    idx = (torch.arange(Lx, device=u.device) - Lx // 2) % Nx
    return z[idx][:, :H]


def _linear(f, g, dims):
    """Linear convolution along dims, the first entries of each axis."""
    N = [_smooth(2 * f.shape[d] - 1) for d in dims]
    if f.is_complex():
        h = torch.fft.ifftn(torch.fft.fftn(f, N, dims) *
                            torch.fft.fftn(g, N, dims), dim=dims)
    else:
        h = torch.fft.irfftn(torch.fft.rfftn(f, N, dims) *
                             torch.fft.rfftn(g, N, dims), N, dims)
    for d in dims:
        h = h.narrow(d, 0, f.shape[d])
    return h.contiguous()


def _centered(f, g, dims):
    """Convolution of centred data (origin at L // 2 of each axis)."""
    F = []
    N = [_smooth(_padded(CENTERED, f.shape[d])) for d in dims]
    idx = [(torch.arange(f.shape[d], device=f.device) - f.shape[d] // 2) % n
           for d, n in zip(dims, N)]
    for z in (f, g):
        for d, n, i in zip(dims, N, idx):
            shape = list(z.shape)
            shape[d] = n
            w = torch.zeros(shape, dtype=z.dtype, device=z.device)
            z = w.index_copy(d, i, z)
        F.append(torch.fft.fftn(z, dim=dims))
    h = torch.fft.ifftn(F[0] * F[1], dim=dims)
    for d, i in zip(dims, idx):
        h = h.index_select(d, i)
    return h


def exact(case, seed):
    family = case["family"]
    if family == "uneven":
        Ls = _lengths(case)
        g = _generator(seed)
        a, b = (_uniform([sum(Ls)], case, g).to(torch.complex128)
                for _ in range(2))
        out, at = torch.empty_like(a), 0
        for n in Ls:
            N = 1 << (2 * n - 1).bit_length()
            out[at:at + n] = torch.fft.ifft(
                torch.fft.fft(a[at:at + n], N) *
                torch.fft.fft(b[at:at + n], N))[:n]
            at += n
        return [out]
    if family == "grad":
        Lx, Ly = case["Lx"], case["Ly"]
        H = (Ly + 1) // 2
        Nx, Ny = (_smooth(_padded(CENTERED, n) + 1) for n in (Lx, Ly))
        while Ny % 2:
            Ny = _smooth(Ny + 1)
        psi, omega = (f.to(torch.complex128).requires_grad_(True)
                      for f in _spectra(case, seed))
        kx = 1j * (torch.arange(Lx, device="cuda", dtype=torch.float64) -
                   Lx // 2)[:, None]
        ky = 1j * torch.arange(H, device="cuda", dtype=torch.float64)[None, :]
        u = [_hermitian_grid(a, Nx, Ny)
             for a in (kx * psi, ky * psi, kx * omega, ky * omega)]
        J = _hermitian_modes(u[0] * u[3] - u[1] * u[2], Lx, H)
        loss = (J.real ** 2 + J.imag ** 2).sum()
        gp, go = torch.autograd.grad(loss, (psi, omega))
        return [loss.detach(), gp, go]
    kinds, L = _axes(case)
    f, g = (x.to(torch.float64 if kinds[0] == REAL else torch.complex128)
            for x in _fields(case, seed))
    if kinds[-1] == HERMITIAN:
        Nx, Ny = (_smooth(_padded(CENTERED, n) + 1) for n in L)
        while Ny % 2:
            Ny = _smooth(Ny + 1)
        h = _hermitian_modes(_hermitian_grid(f, Nx, Ny) *
                             _hermitian_grid(g, Nx, Ny), *f.shape)
        return [h.cpu() if family == "host" else h]
    dims = [d - len(L) for d in range(len(L))]
    return [(_centered if kinds[0] == CENTERED else _linear)(f, g, dims)]
