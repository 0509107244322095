"""LPT stages (csrc/pmx_lpt.cu) against float64 torch: displacements, velocities, the modes'
gradient and the gradient of the gradient, for both orders, odd and even grids and every memory
form of the modes."""

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GRIDS = [(8, 8, 8), (16, 12, 20), (15, 9, 21), (7, 10, 1), (2, 3, 4), (33, 65, 31)]
# float32 transforms of <= 2^17 points: a few ulp (6e-8) times sqrt(17 levels), four of them in a
# row and as many again in the gradient
TOL, GTOL = 2e-6, 4e-6


def _reference(modes, fac, conf):
    shape = conf.ptcl_grid_shape
    kv = []
    for a, n in enumerate(shape):
        f = np.fft.rfftfreq(n) if a == 2 else np.fft.fftfreq(n)
        kv.append(torch.from_numpy(2 * math.pi / conf.ptcl_spacing * f).to(modes.device)
                  .reshape((1,) * a + (-1,) + (1,) * (2 - a)))
    nyq = math.pi / conf.ptcl_spacing
    kz = [torch.where((k.abs() - nyq).abs() < 1e-6 * nyq, 0.0, k) for k in kv]
    k2 = sum(k * k for k in kv)
    inv = torch.where(k2 > 0, -1 / torch.where(k2 > 0, k2, 1.0), 0.0)
    pot = [modes / conf.ptcl_cell_vol * inv]
    if conf.lpt_order > 1:
        phi = {}
        for i in range(3):
            for j in range(i, 3):
                a, b = (kv[i], kv[j]) if i == j else (kz[i], kz[j])
                phi[i, j] = torch.fft.irfftn(-a * b * pot[0], s=shape)
        src = (phi[0, 0] * phi[1, 1] + phi[0, 0] * phi[2, 2] + phi[1, 1] * phi[2, 2]
               - phi[0, 1] ** 2 - phi[0, 2] ** 2 - phi[1, 2] ** 2)
        pot.append(torch.fft.rfftn(src) * inv)
    disp = vel = 0
    for o, p in enumerate(pot):
        g = torch.stack([torch.fft.irfftn(-1j * k * p, s=shape).reshape(-1) for k in kz], dim=1)
        disp, vel = disp + float(fac[o][0]) * g, vel + float(fac[o][1]) * g
    return disp, vel


def _rel(a, b):
    return float((a.detach() - b.detach()).norm() / b.detach().norm())


def _setup(grid, order, seed=2):
    import pmwd_gb300 as pg
    conf = pg.Configuration(1.7, grid, mesh_shape=2, lpt_order=order)
    cosmo = pg.boltzmann(pg.SimpleLCDM(conf), conf, transfer=False, varlin=False)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(seed)
    noise = torch.randn(grid, generator=gen, device='cuda')
    return conf, cosmo, (30 * torch.fft.rfftn(noise)).contiguous(), gen


@pytest.mark.parametrize('order', [1, 2])
@pytest.mark.parametrize('grid', GRIDS)
def test_lpt_and_gradient_against_float64(grid, order):
    import pmwd_gb300 as pg
    from pmwd_gb300 import _hostmath
    conf, cosmo, modes, gen = _setup(grid, order)
    fac = _hostmath.lpt_factors(cosmo, conf)
    lattice = pg.Particles.gen_grid(conf)
    m32 = modes.clone().requires_grad_()
    ptcl, _ = pg.lpt(m32, cosmo, conf)
    m64 = modes.to(torch.complex128).requires_grad_()
    disp, vel = _reference(m64, fac, conf)
    assert torch.equal(ptcl.pmid, lattice.pmid)
    assert _rel(ptcl.vel, vel) < TOL
    assert _rel(ptcl.disp - lattice.disp, disp) < TOL + 2e-7 * float(
        (lattice.disp.norm() + disp.detach().norm()) / disp.detach().norm())
    cots = [torch.randn(disp.shape, generator=gen, device='cuda') for _ in range(2)]
    (got,) = torch.autograd.grad((ptcl.disp, ptcl.vel), m32, cots)
    (want,) = torch.autograd.grad((disp, vel), m64, [c.double() for c in cots])
    assert _rel(got, want) < GTOL
    # one of the outputs alone
    (got,) = torch.autograd.grad(pg.lpt(m32, cosmo, conf)[0].vel, m32, cots[1])
    (want,) = torch.autograd.grad(_reference(m64, fac, conf)[1], m64, cots[1].double())
    assert _rel(got, want) < GTOL


def test_memory_forms_and_graph_give_the_same():
    import pmwd_gb300 as pg
    conf, cosmo, modes, _ = _setup((16, 12, 20), 2)
    ref = pg.lpt(modes.clone().requires_grad_(), cosmo, conf)[0]
    forms = [modes, modes.conj().resolve_conj().conj(),
             modes.permute(2, 0, 1).contiguous().permute(1, 2, 0)]
    for m in forms:
        for grad in (False, True):
            p, _ = pg.lpt(m.detach().requires_grad_() if grad else m, cosmo, conf)
            assert torch.equal(p.disp, ref.disp) and torch.equal(p.vel, ref.vel)


def test_second_derivative():
    """Gradient of a function of the gradient, as the torch operations give it."""
    import pmwd_gb300 as pg
    from pmwd_gb300 import _hostmath
    conf, cosmo, modes, gen = _setup((8, 10, 6), 2)
    fac = _hostmath.lpt_factors(cosmo, conf)
    w = torch.randn((480, 3), generator=gen, device='cuda')

    def second(m, f):
        (g,) = torch.autograd.grad((f(m)[0] ** 2 * w.to(m.real.dtype)).sum(), m, create_graph=True)
        return torch.autograd.grad((g.real ** 2 + g.imag ** 2).sum(), m)[0]

    got = second(modes.clone().requires_grad_(),
                 lambda m: (lambda p: (p.disp - pg.Particles.gen_grid(conf).disp, p.vel))(
                     pg.lpt(m, cosmo, conf)[0]))
    want = second(modes.to(torch.complex128).requires_grad_(), lambda m: _reference(m, fac, conf))
    assert _rel(got, want) < 2e-5


@pytest.mark.parametrize('order', [1, 2])
@pytest.mark.parametrize('grid', [(192, 128, 96), (64, 256, 192), (384, 96, 64), (96, 64, 512)])
def test_own_transforms_against_float64(grid, order):
    """Grids above the graphs' limit whose axes the library transforms itself.  Up to 22
    levels instead of 17: TOL sqrt(22 / 17) = 2.3e-6."""
    import pmwd_gb300 as pg
    from pmwd_gb300 import _hostmath
    conf, cosmo, modes, _ = _setup(grid, order)
    lattice = pg.Particles.gen_grid(conf)
    ptcl, _ = pg.lpt(modes, cosmo, conf)
    disp, vel = _reference(modes.to(torch.complex128), _hostmath.lpt_factors(cosmo, conf), conf)
    assert torch.equal(ptcl.pmid, lattice.pmid)
    assert _rel(ptcl.vel, vel) < 2.3e-6
    assert _rel(ptcl.disp - lattice.disp, disp) < 2.3e-6 + 2e-7 * float(
        (lattice.disp.norm() + disp.norm()) / disp.norm())
