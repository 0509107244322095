"""Particle passes of the force against float64 torch: every deposit mode
(joined lanes at one cell per particle, 8-byte pairs on finer even meshes,
scalar on finer odd ones), periodic wrapping beyond one box length, and cell
sizes with and without an exact reciprocal."""

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [((16, 12, 20), 1, 1.0), ((16, 12, 20), 2, 1.0), ((15, 9, 21), 1, 1.0),
         ((15, 9, 21), 3, 0.7), ((16, 16, 16), 2, 0.3), ((8, 8, 33), 1, 2.0)]


def _cic(x, shape):
    lo = torch.floor(x)
    for k in range(8):
        idx, w = 0, 1
        for a in range(3):
            b = k >> a & 1
            f = x[:, a] - lo[:, a]
            idx = idx * shape[a] + torch.remainder(lo[:, a] + b, shape[a]).long()
            w = w * (f if b else 1 - f)
        yield idx, w


def _accelerations(x, shape, cell, per):
    dens = torch.zeros(shape, dtype=torch.float64, device=x.device).reshape(-1)
    for i, w in _cic(x, shape):
        dens = dens.index_add(0, i, w * per)
    kv = [2 * math.pi / cell * torch.from_numpy(f).to(x.device).reshape((1,) * a + (-1,) + (1,) * (2 - a))
          for a, f in enumerate([np.fft.fftfreq(shape[0]), np.fft.fftfreq(shape[1]),
                                 np.fft.rfftfreq(shape[2])])]
    k2 = sum(k * k for k in kv)
    inv = torch.where(k2 > 0, -1.5 * 0.3 / torch.where(k2 > 0, k2, 1.0), 0.0)
    pot = torch.fft.rfftn(dens.reshape(shape)) * inv
    acc = []
    for k in kv:
        k = torch.where((k.abs() - math.pi / cell).abs() < 1e-6 / cell, 0.0, k)
        m = torch.fft.irfftn(-1j * k * pot, s=shape).reshape(-1)
        acc.append(sum(m[i] * w for i, w in _cic(x, shape)))
    return torch.stack(acc, dim=1)


@pytest.mark.parametrize('grid,ratio,spacing', CASES)
@pytest.mark.parametrize('state', ['wave', 'spread', 'one cell'])
def test_force_and_vjp_against_float64(grid, ratio, spacing, state):
    import pmwd_gb300 as pg
    conf = pg.Configuration(spacing, grid, mesh_shape=ratio)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(6)
    p = pg.Particles.gen_grid(conf)
    rnd = torch.randn(p.disp.shape, generator=gen, device='cuda')
    cell = conf.cell_size
    if state == 'wave':       # neighbours stay in order; the overdensity is of order one half
        box = torch.tensor(conf.box_size, device='cuda')
        q = p.pmid.float() * cell + p.disp
        disp = p.disp + 0.31 * cell + 0.08 * box * torch.sin(2 * math.pi * q / box)
    elif state == 'spread':   # up to several box lengths away, on both sides
        disp = p.disp + 0.4 * max(conf.box_size) * rnd
    else:                     # every second particle into one cell
        pos = p.pmid.float() * cell
        target = torch.full_like(pos, 2.4 * cell) + 0.1 * cell * rnd
        disp = torch.where((torch.arange(len(p), device='cuda') % 2 == 0)[:, None], target - pos,
                           p.disp + 0.37 * cell)
    disp = disp.contiguous().requires_grad_()
    cosmo = pg.SimpleLCDM(conf)
    acc = pg.gravity(0.5, p.replace(disp=disp), cosmo, conf)
    cot = torch.randn(acc.shape, generator=gen, device='cuda')
    (got,) = torch.autograd.grad(acc, disp, cot)
    # x = disp / cell in float32, as the package defines the fractions
    x32 = (disp.detach() / torch.tensor(cell, dtype=torch.float32, device='cuda')).double()
    x = (p.pmid.double() + x32).requires_grad_()
    want = _accelerations(x, tuple(conf.mesh_shape), cell, conf.mesh_size / conf.ptcl_num)
    (gx,) = torch.autograd.grad(want, x, cot.double())
    # fractions carry the ulp of x (2^-24 |x|), sums of 8 to n terms and a float32 transform
    # some ulp more
    tol = 2e-6 + 4 * 2 ** -24 * float(x32.abs().max())
    assert float((acc - want).detach().norm() / want.detach().norm()) < tol
    assert float((got - gx / cell).norm() / (gx / cell).norm()) < 10 * tol
