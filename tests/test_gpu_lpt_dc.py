"""The k = 0 mode does not enter the displacements (lpt.py:30-34, gravity.py:9-16 set its potential
to zero), whatever its value: a spectrum such as 1 / k leaves an infinity there."""

import math

import pytest
import torch

import pmwd_gb300 as pg

pytestmark = pytest.mark.gpu


# replayed graph, own transforms, and with a gradient the stages between torch's transforms
@pytest.mark.parametrize('grid, grad', [((12, 10, 9), False), ((192, 128, 96), False),
                                        ((130, 128, 140), False), ((12, 10, 9), True)])
@pytest.mark.parametrize('order', [1, 2])
@pytest.mark.parametrize('dc', [math.inf, math.nan])
def test_zero_mode_is_ignored(cuda, grid, grad, order, dc):
    conf = pg.Configuration(1.7, grid, mesh_shape=1, lpt_order=order)
    cosmo = pg.boltzmann(pg.SimpleLCDM(conf), conf, transfer=False, varlin=False)
    gen = torch.Generator(device=cuda).manual_seed(8)
    modes = (30 * torch.fft.rfftn(torch.randn(grid, generator=gen, device=cuda))).contiguous()
    out = []
    for value in (0.0, dc):
        m = modes.clone()
        m[0, 0, 0] = value
        m.requires_grad_(grad)
        p, _ = pg.lpt(m, cosmo, conf)
        out.append([p.disp.detach(), p.vel.detach()])
        if grad:
            out[-1].append(torch.autograd.grad((p.disp.square().sum(), p.vel.sum()), m)[0])
    for a, b in zip(*out):
        assert torch.equal(a, b)
