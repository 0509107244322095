"""Meshes whose first axis is a power of two and whose others the library's own transforms do
not have: slab-wise 2-D cuFFT planes and the fused x pass (of 64, 128 and 256 points), with one
and several slabs per component, one to three chains, replayed as graphs and issued directly,
single and batched.  And batches of meshes on the own transforms whose first axis is not a
power of two."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import cosmo as oc, pm
from pmwd_gb300 import _lib
from test_gpu_batch import batch_run, close_cot, make_sim, rel, single_run
from test_gpu_force import RTOL_ACC, make, rel_l2

pytestmark = pytest.mark.gpu

# particle grid, mesh factor: meshes (64, 80, 80), (128, 48, 160), (256, 160, 160)
SHAPES = [((16, 20, 20), 4), ((32, 12, 40), 4), ((64, 40, 40), 4)]
VARIANTS = [{}, {'slab_log2': 2, 'chains': 1}, {'slab_log2': 1, 'chains': 3},
            {'slab_log2': 3, 'graphs': False}]


@pytest.mark.parametrize('ptcl, ratio', SHAPES)
def test_force_and_vjp_match_oracle(cuda, ptcl, ratio):
    oconf, gconf, pmid, disp, _ = make(ptcl, ratio, 1.0, 1.5)
    cot = np.random.default_rng(3).normal(size=disp.shape).astype(np.float32)
    oconf64 = oc.OConf(1.0, ptcl, ratio, float_dtype=np.float64)
    acc_o, dc_o, om_o = pm.gravity_vjp(pmid, disp.astype(np.float64), 0.3, oconf64,
                                       cot.astype(np.float64))
    P, D, C = (torch.from_numpy(np.ascontiguousarray(x)).to(cuda) for x in (pmid, disp, cot))
    spec = _lib.make_spec(3, gconf.mesh_shape, gconf.mesh_shape, gconf.cell_size)
    st = _lib.stream_ptr(cuda)
    for kw in VARIANTS:
        ws = _lib.Workspace(gconf.mesh_shape, adjoint=True, **kw)
        for _ in range(2):   # the second call replays the graphs that the first one captured
            f, a, dc = (torch.empty_like(D) for _ in range(3))
            om = torch.zeros((), dtype=torch.float64, device=cuda)
            _lib.call('pmx_force', ws.handle, spec, P, D, len(P), gconf.ptcl_num, 0.3, f, st)
            _lib.call('pmx_force_vjp', ws.handle, spec, P, D, len(P), gconf.ptcl_num, 0.3, C, a, dc,
                      om, st)
            for x in (f, a):
                assert rel_l2(x.cpu().numpy(), acc_o) < RTOL_ACC, kw
            assert rel_l2(dc.cpu().numpy(), dc_o) < 1e-4, kw
            assert abs(float(om) / om_o - 1) < 1e-4, kw
        del ws


@pytest.mark.parametrize('kw', VARIANTS[:2])
@pytest.mark.parametrize('ptcl, ratio', SHAPES)
def test_multistep_equals_single_steps(cuda, ptcl, ratio, kw):
    """Steps in one call against the same steps one by one: only the order of the float32
    reductions differs."""
    k = 4
    sim = make_sim(cuda, ptcl, ratio, float(ratio), 4, 0.3, k)
    conf, n = sim['conf'], len(sim['pmid'])
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    st = _lib.stream_ptr(cuda)
    out = []
    for multi in (False, True):
        ws = _lib.Workspace(conf.mesh_shape, adjoint=False, **kw)
        d, v = sim['disp'].clone(), sim['vel'].clone()
        a = torch.empty_like(d)
        _lib.call('pmx_force', ws.handle, spec, sim['pmid'], d, n, conf.ptcl_num, 0.3, a, st)
        if multi:
            _lib.call('pmx_nbody_steps', ws.handle, spec, sim['pmid'], d, v, a, n, conf.ptcl_num, k,
                      sim['fac'].ctypes.data_as(ctypes.c_void_p), 0.3, st)
        else:
            for f in sim['fac']:
                _lib.call('pmx_nbody_step', ws.handle, spec, sim['pmid'], d, v, a, n, conf.ptcl_num,
                          (_lib.c_f * 3)(*f), 0.3, st)
        out.append((d, v, a))
    for x, y in zip(*out):
        assert rel(y, x) < 1e-5


@pytest.mark.parametrize('mesh, chunks', [((64, 80, 80), None), ((128, 48, 160), [2, 3]),
                                          ((96, 64, 128), [1, 4])])
def test_batch_equals_single(cuda, mesh, chunks):
    """As the batched test of the cubic meshes: two particle grids of one mesh, bounds and all."""
    k = 5
    half = tuple(n // 2 for n in mesh)
    sims = [make_sim(cuda, half, 2, 2.0, 1, 0.3, k), make_sim(cuda, mesh, 1, 1.0, 2, 0.25, k),
            make_sim(cuda, half, 2, 2.0, 3, 0.35, k)]
    bf, ba = batch_run(sims, k, cuda, chunks)
    for s, bfi, bai in zip(sims, bf, ba):
        sf, sa = single_run(s, k, cuda)
        for a, b in zip(bfi, sf):
            assert rel(a, b) < 1e-5
        for a, b in zip(bai[:3], sa[:3]):
            assert rel(a, b) < 1e-4
        for a, b in zip(bai[3:6], sa[3:6]):
            assert close_cot(a, b)
        np.testing.assert_allclose(bai[6].cpu().numpy(), sa[6].cpu().numpy(), rtol=3e-3,
                                   atol=1e-5 * float(sa[6].abs().max()))
