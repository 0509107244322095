"""Default-enmesh scatter and gather (k_*_cic) and their VJPs against float64 torch, over channels,
mesh ratios (joined and paired reductions), odd sizes, meshes larger than the periodic box,
unaligned meshes and particles far outside the box."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cic(x, wrap, shape):
    lo = torch.floor(x.detach())
    for k in range(8):
        idx, w = 0, 1
        for a in range(3):
            b = k >> a & 1
            f = x[:, a] - lo[:, a]
            idx = idx * shape[a] + torch.remainder(lo[:, a] + b, wrap[a]).long()
            w = w * (f if b else 1 - f)
        yield idx, w


def _rel(a, b):
    return float((a.detach().double() - b.detach()).norm() / b.detach().norm())


@pytest.mark.parametrize('extra', [0, 3])
@pytest.mark.parametrize('chan', [0, 1, 3])
@pytest.mark.parametrize('grid,ratio', [((16, 12, 20), 1), ((8, 6, 10), 2), ((15, 9, 33), 1),
                                        ((5, 3, 7), 3), ((2, 2, 2), 1)])
@pytest.mark.parametrize('far', [False, True])
def test_scatter_gather_against_float64(grid, ratio, chan, extra, far):
    import pmwd_gb300 as pg
    from pmwd_gb300 import _lib
    conf = pg.Configuration(0.9, grid, mesh_shape=ratio)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(8)
    rand = lambda *s: torch.randn(s, generator=gen, device='cuda')
    p = pg.Particles.gen_grid(conf)
    n, cell, nc = len(p), conf.cell_size, max(chan, 1)
    disp = (p.disp + (40 if far else 0.3) * cell * rand(n, 3)).contiguous().requires_grad_()
    shape = tuple(m + extra for m in conf.mesh_shape)
    cs = (chan,) if chan else ()
    x32 = (disp.detach() / torch.tensor(cell, dtype=torch.float32, device='cuda')).double()
    x = (p.pmid.double() + x32).requires_grad_()
    nb = list(_cic(x, conf.mesh_shape, shape))
    ptcl = p.replace(disp=disp)
    tol = 1e-6 + 4 * 2 ** -24 * float(x32.abs().max())   # the fractions carry the ulp of x

    # scatter
    val = rand(n, *cs).requires_grad_() if chan else None
    start = rand(*shape, *cs)
    mesh = pg.scatter(ptcl, conf, mesh=start, val=val)
    v64 = (val.detach().double() if chan else torch.full((n,), conf.mesh_size / conf.ptcl_num,
           dtype=torch.float64, device='cuda')).reshape(n, nc).requires_grad_()
    want = start.double().reshape(-1, nc)
    for i, w in nb:
        want = want.index_add(0, i, w[:, None] * v64)
    assert _rel(mesh, want.reshape(mesh.shape)) < tol
    cot = rand(*mesh.shape)
    ins = [disp] + ([val] if chan else [])
    got = torch.autograd.grad(mesh, ins, cot)
    ref = torch.autograd.grad(want, [x, v64], cot.double().reshape(-1, nc), retain_graph=True)
    assert _rel(got[0], ref[0] / cell) < 4 * tol
    if chan:
        assert _rel(got[1], ref[1].reshape(val.shape)) < 4 * tol
    if not extra:   # the default mesh: the same without the start
        fresh = pg.scatter(ptcl, conf, val=val)
        assert _rel(fresh, (want - start.double().reshape(-1, nc)).reshape(mesh.shape)) < 4 * tol

    # gather
    m = rand(*shape, *cs).requires_grad_()
    add = rand(n, *cs)
    out = pg.gather(ptcl, conf, m, val=add)
    m64 = m.detach().double().reshape(-1, nc).requires_grad_()
    want = add.double().reshape(n, nc) + sum(m64[i] * w[:, None] for i, w in nb)
    assert _rel(out, want.reshape(out.shape)) < tol
    cot = rand(*out.shape)
    got = torch.autograd.grad(out, [disp, m], cot)
    ref = torch.autograd.grad(want, [x, m64], cot.double().reshape(n, nc))
    assert _rel(got[0], ref[0] / cell) < 4 * tol
    assert _rel(got[1], ref[1].reshape(m.shape)) < 4 * tol

    # an array that starts 4 bytes off an 8-byte boundary
    buf = torch.zeros(int(np.prod(shape)) * nc + 1, device='cuda')
    spec = _lib.make_spec(3, conf.mesh_shape, shape, cell)
    vals = rand(n, nc)
    _lib.call('pmx_scatter', spec, p.pmid, disp.detach(), n, vals, 0.0, nc, buf[1:],
              _lib.stream_ptr())
    want = torch.zeros((int(np.prod(shape)), nc), dtype=torch.float64, device='cuda')
    for i, w in nb:
        want = want.index_add(0, i, w.detach()[:, None] * vals.double())
    assert _rel(buf[1:].reshape(-1, nc), want) < tol and float(buf[0]) == 0
