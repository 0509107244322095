"""Mesh transforms of the Poisson solve (csrc/pmx_mesh_fft.cuh) against 3-D
cuFFT plans of the same library: the force, its VJP and the Omega_m term."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# every supported axis length, on each axis, and mixed boxes
SHAPES = ([(n, 64, 96) for n in (96, 128, 192, 256, 384, 512, 768, 1024)]
          + [(64, n, 96) for n in (96, 128, 192, 256, 384, 512, 768, 1024)]
          + [(96, 64, n) for n in (64, 96, 128, 192, 256, 384, 512, 768, 1024)]
          + [(128, 128, 128), (384, 192, 96)])


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize('shape', SHAPES)
def test_force_and_vjp_against_cufft(shape):
    import pmwd_gb300 as pg
    from pmwd_gb300 import _lib
    grid = tuple(n // 2 for n in shape)
    conf = pg.Configuration(1.0, grid, mesh_shape=2)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(3)
    p = pg.Particles.gen_grid(conf)
    disp = p.disp + 0.7 * torch.randn(p.disp.shape, generator=gen, device='cuda')
    cot = torch.randn(p.disp.shape, generator=gen, device='cuda')
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    res = []
    for kw in ({}, {'cufft3d': True}):
        ws = _lib.Workspace(conf.mesh_shape, **kw)
        acc, dcot = torch.empty_like(disp), torch.empty_like(disp)
        om = torch.empty((), dtype=torch.float64, device='cuda')
        _lib.call('pmx_force_vjp', ws.handle, spec, p.pmid, disp, disp.shape[0], conf.ptcl_num,
                  0.3, cot, acc, dcot, om, _lib.stream_ptr())
        torch.cuda.synchronize()
        res.append((acc, dcot, float(om)))
    # two float32 transforms of log2(M) <= 30 levels each differ by a few ulp (6e-8) per
    # sqrt(level): 2 * 6e-8 * sqrt(30) * 2 transforms = 1.3e-6; the VJP runs twice as many
    assert _rel(res[0][0], res[1][0]) < 1.3e-6
    assert _rel(res[0][1], res[1][1]) < 2.6e-6
    # the Omega_m term is sum(cot . acc) of random signs: its error is that of acc times the
    # norms, not relative to the (cancelling) sum
    scale = float(cot.norm() * res[1][0].norm()) / 0.3
    assert abs(res[0][2] - res[1][2]) < 1.3e-6 * scale


@pytest.mark.parametrize('shape', ((64, 64, 64), (256, 64, 64), (64, 96, 96), (96, 128, 128),
                                   (128, 192, 192)))
def test_square_planes(shape):
    """n x n planes: z and y axes in one kernel up to n = 128, two beyond."""
    test_force_and_vjp_against_cufft(shape)


def test_batched_equals_single():
    """Two slots of one batched call against two single-simulation forces: one x-axis launch
    serves both with its own Green's constant."""
    import ctypes

    import pmwd_gb300 as pg
    from pmwd_gb300 import _lib
    conf = pg.Configuration(1.0, (48, 32, 64), mesh_shape=2)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(4)
    p = pg.Particles.gen_grid(conf)
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    n = len(p)
    oms, disps = (0.25, 0.4), [p.disp + torch.randn(p.disp.shape, generator=gen, device='cuda')
                               for _ in range(2)]
    single = _lib.Workspace(conf.mesh_shape)
    want = []
    for om, d in zip(oms, disps):
        acc = torch.empty_like(d)
        _lib.call('pmx_force', single.handle, spec, p.pmid, d, n, conf.ptcl_num, om, acc,
                  _lib.stream_ptr())
        want.append(acc)
    ws = _lib.Workspace(conf.mesh_shape, slots=2)
    sims = (_lib.PmxSim * 2)()
    got, vel = [torch.empty_like(d) for d in disps], [torch.zeros_like(d) for d in disps]
    for b in range(2):
        s = sims[b]
        s.pmid, s.disp, s.vel, s.acc = (t.data_ptr() for t in (p.pmid, disps[b], vel[b], got[b]))
        s.n, s.ptcl_num, s.omega_m = n, conf.ptcl_num, oms[b]
    _lib.check(_lib.load().pmx_nbody_steps_batch(ws.handle, spec, 2, sims, 1, 0,
                                                 _lib.stream_ptr()), 'pmx_nbody_steps_batch')
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert _rel(a, b) < 1e-6   # the order of the float32 deposits differs


@pytest.mark.parametrize('shape', ((64, 64, 64), (128, 192, 192)))
def test_captured_steps_replay(shape):
    """Multi-step calls under stream capture, between copies: the kernels' programmatic
    launches become graph edges.  The deposits' order differs, as between two runs."""
    import pmwd_gb300 as pg
    from pmwd_gb300 import _lib
    conf = pg.Configuration(1.0, tuple(n // 2 for n in shape), mesh_shape=2)
    gen = torch.Generator(device='cuda')
    gen.manual_seed(5)
    p = pg.Particles.gen_grid(conf)
    start = p.disp + 0.3 * torch.randn(p.disp.shape, generator=gen, device='cuda')
    disp, vel, acc = start.clone(), torch.zeros_like(start), torch.zeros_like(start)
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    ws = _lib.Workspace(conf.mesh_shape)
    fac = (_lib.c_f * 9)(*(0.01, 0.02, 0.01) * 3)
    out = torch.empty_like(start)

    def run():
        disp.copy_(start)
        vel.zero_()
        acc.zero_()
        _lib.call('pmx_force', ws.handle, spec, p.pmid, disp, len(p), conf.ptcl_num, 0.3, acc,
                  _lib.stream_ptr())
        _lib.call('pmx_nbody_steps', ws.handle, spec, p.pmid, disp, vel, acc, len(p),
                  conf.ptcl_num, 3, fac, 0.3, _lib.stream_ptr())
        out.copy_(vel)

    run()
    want = out.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run()
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert _rel(out, want) < 1e-6   # the order of the float32 deposits differs
