"""Forms in which torch asks lpt for the modes' gradient besides one plain backward call."""

import pytest
import torch

import pmwd_gb300 as pg

pytestmark = pytest.mark.gpu

# float32 transforms in another order: as the stages' own gradient test
GTOL = 4e-6


def _setup(cuda, order=2, grid=(6, 9, 8)):
    conf = pg.Configuration(1.7, grid, mesh_shape=1, lpt_order=order)
    cosmo = pg.boltzmann(pg.SimpleLCDM(conf), conf, transfer=False, varlin=False)
    gen = torch.Generator(device=cuda).manual_seed(5)
    modes = (30 * torch.fft.rfftn(torch.randn(grid, generator=gen, device=cuda))).contiguous()
    cots = torch.randn((3, conf.ptcl_num, 3), generator=gen, device=cuda)
    return conf, cosmo, modes, cots


def _close(a, b):
    assert a.shape == b.shape
    assert float((a - b).norm() / b.norm()) < GTOL


@pytest.mark.parametrize('order', [1, 2])
@pytest.mark.parametrize('create', [False, True])
def test_batched_cotangents(cuda, order, create):
    conf, cosmo, modes, cots = _setup(cuda, order)
    m = modes.requires_grad_()
    p, _ = pg.lpt(m, cosmo, conf)
    want = torch.stack([torch.autograd.grad((p.disp, p.vel), m, (c, 2 * c), retain_graph=True)[0]
                        for c in cots])
    (got,) = torch.autograd.grad((p.disp, p.vel), m, (cots, 2 * cots), is_grads_batched=True,
                                 retain_graph=True, create_graph=create)
    _close(got.detach(), want)
    got = torch.vmap(lambda c: torch.autograd.grad((p.disp, p.vel), m, (c, 2 * c), retain_graph=True,
                                                   create_graph=create)[0])(cots)
    _close(got.detach(), want)
    # one of the outputs alone
    want = torch.stack([torch.autograd.grad(p.vel, m, c, retain_graph=True)[0] for c in cots])
    (got,) = torch.autograd.grad(p.vel, m, cots, is_grads_batched=True)
    _close(got, want)


def test_vectorised_jacobian(cuda):
    conf, cosmo, modes, _ = _setup(cuda, grid=(4, 3, 2))

    def f(x):
        return pg.lpt(torch.view_as_complex(x), cosmo, conf)[0].disp

    x = torch.view_as_real(modes).clone()
    _close(torch.autograd.functional.jacobian(f, x, vectorize=True),
           torch.autograd.functional.jacobian(f, x))


@pytest.mark.parametrize('grad', [False, True])
def test_negative_views(cuda, grad):
    """Modes and cotangents whose sign is still to be applied (torch's negative bit)."""
    conf, cosmo, modes, cots = _setup(cuda)
    view = torch._neg_view(modes)
    assert view.is_neg() and view.is_contiguous()
    got = pg.lpt(view.detach().requires_grad_(grad), cosmo, conf)[0]
    want = pg.lpt((-modes).requires_grad_(grad), cosmo, conf)[0]
    assert torch.equal(got.vel, want.vel)
    if grad:
        m = modes.clone().requires_grad_()
        out = pg.lpt(m, cosmo, conf)[0].disp
        (got,) = torch.autograd.grad(out, m, torch._neg_view(cots[0]), retain_graph=True)
        (want,) = torch.autograd.grad(out, m, -cots[0])
        assert torch.equal(got, want)


@pytest.mark.parametrize('order', [1, 2])
def test_modes_changed_in_place_before_backward(cuda, order):
    """The gradient is that of the call's modes, whatever their owner does with them after it;
    a gradient that would have to read them again is refused."""
    conf, cosmo, modes, cots = _setup(cuda, order)
    m = modes.clone().requires_grad_()
    p, _ = pg.lpt(m, cosmo, conf)
    (want,) = torch.autograd.grad((p.disp, p.vel), m, (cots[0], cots[1]), retain_graph=True)
    with torch.no_grad():
        m.mul_(-3)
    (got,) = torch.autograd.grad((p.disp, p.vel), m, (cots[0], cots[1]), retain_graph=True)
    assert torch.equal(got, want)
    with pytest.raises(RuntimeError, match='modified by an inplace operation'):
        torch.autograd.grad(p.disp, m, cots[0], create_graph=True)
