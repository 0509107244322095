"""A batch of simulations with different particle densities deposits each of them as it is
deposited alone.  Particles sit on the lattice but for a step of 2^-24 of a cell along z, one
particle per cell: a cell's density is 1 - s of its own and s' of its lower neighbour's
particle.  Added one after the other to the mesh's -1, all sums are exact; added to each other
first, as lanes that join their neighbour's value do, 1 - s + s' rounds where it exceeds 1.  So
the density, and with it every bit of the accelerations, tells the two apart, whatever the order
of the reductions."""

import pytest
import torch

import pmwd_gb300 as pg
from pmwd_gb300 import _lib

pytestmark = pytest.mark.gpu


def _sim(cuda, side, ratio, seed):
    conf = pg.Configuration(float(ratio), (side,) * 3, ratio)   # cell size 1
    p = pg.Particles.gen_grid(conf, device=cuda)
    gen = torch.Generator(device=cuda).manual_seed(seed)
    disp = torch.zeros_like(p.disp)
    disp[:, 2] = 2.0 ** -24 * torch.randint(0, 64, (len(disp),), generator=gen, device=cuda)
    return conf, p.pmid, disp


def _batch(cuda, sims):
    conf = sims[0][0]
    ws = _lib.Workspace(conf.mesh_shape, adjoint=False, slots=len(sims))
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    arr = (_lib.PmxSim * len(sims))()
    state = []
    for i, (c, pmid, disp) in enumerate(sims):
        d, v, a = disp.clone(), torch.zeros_like(disp), torch.empty_like(disp)
        state.append((d, v, a))
        arr[i] = _lib.PmxSim(pmid.data_ptr(), d.data_ptr(), v.data_ptr(), a.data_ptr(), None, None,
                             None, len(pmid), c.ptcl_num, 0.3, None, None)
    _lib.call('pmx_nbody_steps_batch', ws.handle, spec, len(sims), arr, 1, 0, _lib.stream_ptr(cuda))
    torch.cuda.synchronize()
    return [a for _, _, a in state]


def _alone(cuda, sim):
    conf, pmid, disp = sim
    ws = _lib.Workspace(conf.mesh_shape, adjoint=False)
    spec = _lib.make_spec(3, conf.mesh_shape, conf.mesh_shape, conf.cell_size)
    acc = torch.empty_like(disp)
    _lib.call('pmx_force', ws.handle, spec, pmid, disp, len(pmid), conf.ptcl_num, 0.3, acc,
              _lib.stream_ptr(cuda))
    torch.cuda.synchronize()
    return acc


@pytest.mark.parametrize('dense_first', [True, False])
def test_mixed_densities_deposit_as_alone(cuda, dense_first):
    dense, sparse = _sim(cuda, 64, 1, 1), _sim(cuda, 32, 2, 2)
    want = _alone(cuda, dense)
    assert float(want.abs().max()) > 0
    sims = [dense, sparse] if dense_first else [sparse, dense]
    got = _batch(cuda, sims)[0 if dense_first else 1]
    assert torch.equal(got, want)
