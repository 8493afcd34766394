"""GPU: the tensors an AdvectionJacobian keeps: usable by autograd however the
operator was made, on any stream, broadcasting as the full grids would, and
held by a captured step."""
import gc

import pytest

pytestmark = pytest.mark.gpu

LX, LY = 31, 47


def _spectra(dtype, seed=7):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((LX, (LY + 1) // 2), generator=g, device="cuda",
                        dtype=dtype) for _ in range(2)]


def _step(op, psi, omega):
    import torch
    psi, omega = (t.detach().clone().requires_grad_(True)
                  for t in (psi, omega))
    J = op(psi, omega)
    loss = (J.real ** 2 + J.imag ** 2).sum()
    return (J.detach(), *torch.autograd.grad(loss, (psi, omega)))


@pytest.mark.parametrize("precision", ["f64", "f32", "ff"])
def test_made_in_inference_mode(native_lib, precision):
    import torch
    from fftwpp_gb300.autograd import AdvectionJacobian, wavenumbers
    with torch.inference_mode():
        op = AdvectionJacobian(LX, LY, precision)
    psi, omega = _spectra(op.dtype)
    got = _step(op, psi, omega)
    kx, ky = wavenumbers(LX, LY, "cuda", op.dtype.to_real())
    a = [w.clone().requires_grad_(True) for w in (psi, omega)]
    J = op.jacobian(1j * kx * a[0], 1j * ky * a[0], 1j * kx * a[1],
                    1j * ky * a[1])
    loss = (J.real ** 2 + J.imag ** 2).sum()
    want = (J.detach(), *torch.autograd.grad(loss, a))
    assert all(torch.equal(x, y) for x, y in zip(got, want))


def test_broadcast_inputs(native_lib):
    """A column or a scalar stands for a whole spectrum, as in a product with
    the full wavenumber grids."""
    import torch
    from fftwpp_gb300.autograd import AdvectionJacobian
    op = AdvectionJacobian(LX, LY)
    psi, omega = _spectra(op.dtype)
    col = psi[:, :1].contiguous()
    for x in (col, psi[:1].contiguous(), psi[:1, :1].contiguous()):
        assert torch.equal(op(x, omega),
                           op(x.expand_as(omega).contiguous(), omega))
    with pytest.raises(RuntimeError):
        op(psi[:, :3].contiguous(), omega)


def test_other_streams(native_lib):
    """Results on side streams equal those on the default one, also when the
    operator is dropped behind them and its memory asked for again."""
    import torch
    from fftwpp_gb300.autograd import AdvectionJacobian
    op = AdvectionJacobian(LX, LY)
    psi, omega = _spectra(op.dtype)
    want = _step(op, psi, omega)
    for _ in range(8):
        op = AdvectionJacobian(LX, LY)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            got = _step(op, psi, omega)
        del op
        gc.collect()
        junk = [torch.full((LX,), 1e30, dtype=psi.dtype, device="cuda")
                for _ in range(64)]
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip(got, want))
        del junk


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_captured_step_holds_its_operator(native_lib, precision):
    import torch
    from fftwpp_gb300.autograd import AdvectionJacobian, GraphedLossStep
    op = AdvectionJacobian(LX, LY, precision)
    psi, omega = _spectra(op.dtype)
    want = _step(op, psi, omega)
    step = GraphedLossStep(op, psi.clone(), omega.clone())
    assert step.op is op
    del op
    gc.collect()
    for _ in range(2):
        _, gp, go = step()
        assert torch.equal(gp, want[1]) and torch.equal(go, want[2])
