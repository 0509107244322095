"""The work that this package is timed on: single forces, N-body runs, their gradients, the mesh
operators, Lagrangian initial conditions and the power spectrum, each through the public API.

A case is a dict of plain values:

* ``kind``     'force', 'nbody', 'scatter', 'gather', 'lpt' or 'powspec';
* ``g0 g1 g2`` the particle grid (the field's grid for 'powspec');
* ``ratio``    mesh cells per particle along each axis;
* ``grad``     also run the backward pass, against given cotangents;
* ``state``    'early' (a = 1/64, displacements of a tenth of a spacing), 'mid' (a = 1/8, nearly a
  spacing), 'late' (a = 1/2, a few spacings) or 'halos' (late, part of the particles collapsed);
* ``steps``    leapfrog steps ('nbody'), ``da`` the scale-factor step;
* ``chan``     channels ('scatter', 'gather'; 0: the default scalar density);
* ``cell``     target cell size in mesh cells ('scatter', 'gather'; 0: the mesh's own), with
  ``offset``, the target mesh's origin in mesh cells;
* ``bins``, ``cross``, ``deconv``  the binning ('log' or 'lin'), a cross spectrum, the window power.

Inputs come from the seed alone: a Gaussian random field with a turnover spectrum gives Zel'dovich
displacements and velocities of the stated amplitude.
"""

import math

import numpy as np
import torch

import pmwd_gb300 as pm
from pmwd_gb300.spec_util import powspec

# scale factor and displacement rms (in spacings) of each state
STATES = {'early': (1 / 64, 0.1), 'mid': (1 / 8, 0.8), 'late': (1 / 2, 2.5), 'halos': (1 / 2, 2.5)}
DA, DA_FINE = 1 / 64, 1 / 512
OMEGA_M = 0.3


def _case(kind, grid, name=None, **kw):
    c = {'kind': kind, 'g0': grid[0], 'g1': grid[1], 'g2': grid[2], 'ratio': 1.0, 'grad': False,
         'state': 'early', 'steps': 0, 'da': DA, 'chan': 0, 'cell': 0.0, 'offset': 0.0, 'bins': 'log',
         'cross': False, 'deconv': 0}
    c.update(kw)
    if name is not None:
        c['name'] = name
    return c


def listed():
    return [
        # one force on the smallest mesh that the published timing table has: launches and latency
        _case('force', (64,) * 3, 'force_64'),
        # a small run (the first quarter, on a 128^3 mesh), as a parameter scan makes by the
        # thousand: per-step launches
        _case('nbody', (64,) * 3, 'nbody_64', ratio=2.0, steps=16),
        # the gradient study of the adjoint paper: 128^3 particles, 256^3 mesh, some of its steps,
        # forward and reversible adjoint with respect to the particles' state
        _case('nbody', (128,) * 3, 'nbody_128_grad', ratio=2.0, steps=5, grad=True, state='mid',
              da=DA_FINE),
        # the quickstart's size in its late, clustered part, forward only
        _case('nbody', (256,) * 3, 'nbody_256_late', ratio=2.0, steps=8, state='late'),
        # the adjoint notebook's grid: not a power of two, one cell per particle
        _case('nbody', (384,) * 3, 'nbody_384', steps=6),
        # the headline workload, 512^3 particles on a 1024^3 mesh, forward and adjoint
        _case('nbody', (512,) * 3, 'nbody_512_grad', ratio=2.0, steps=3, grad=True, state='mid',
              da=DA_FINE),
        # a ragged box (a survey's bounding box), force and its VJP
        _case('force', (90, 75, 60), 'force_ragged_grad', ratio=2.0, grad=True),
        # the density of a clustered snapshot and its VJP: the contended deposit
        _case('scatter', (256,) * 3, 'scatter_halos_grad', state='halos', grad=True),
        # a three-component field read at the particles of an odd-sized grid, and its VJP
        _case('gather', (175, 125, 225), 'gather_3ch_grad', ratio=1.0, state='late', chan=3,
              grad=True),
        # initial conditions of the quickstart's size from linear modes
        _case('lpt', (256,) * 3, 'lpt_256'),
        # differentiable initial conditions, as a field-level fit needs them, on an odd-sized grid
        _case('lpt', (96, 72, 120), 'lpt_96_grad', grad=True),
        # the power spectrum of a density mesh, as analyses bin it
        _case('powspec', (512,) * 3, 'powspec_512', deconv=2),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, lo, hi):
    """A cubic power-of-two grid, a power-of-two box, a cubic grid of any size or any box."""
    u = rng.random()
    if u < 0.4:
        a, b = math.ceil(math.log2(lo)), math.floor(math.log2(hi))
        if u < 0.25:
            return (2 ** rng.randint(a, b),) * 3
        return tuple(2 ** rng.randint(a, b) for _ in range(3))
    if u < 0.7:
        return (_log_uniform(rng, lo, hi),) * 3
    n = _log_uniform(rng, lo, hi)
    return tuple(max(8, min(hi, round(n * rng.uniform(0.6, 1.6)))) for _ in range(3))


def draw(rng):
    known = [{k: v for k, v in c.items() if k != 'name'} for c in listed()]
    while True:
        c = _draw(rng)
        if c not in known:
            return c


def _draw(rng):
    kind = rng.choice(('force', 'nbody', 'nbody', 'scatter', 'gather', 'lpt', 'powspec'))
    if kind == 'powspec':
        return _case(kind, _grid(rng, 32, 512), bins=rng.choice(('log', 'lin')),
                     cross=rng.random() < 0.3, deconv=rng.choice((0, 2)))
    if kind == 'lpt':
        return _case(kind, _grid(rng, 24, 256), grad=rng.random() < 0.5)
    if kind in ('scatter', 'gather'):
        chan = rng.choice((0, 0, 1, 3)) if kind == 'scatter' else rng.choice((1, 3))
        own = rng.random() < 0.7
        return _case(kind, _grid(rng, 24, 256), ratio=rng.choice((1.0, 2.0)),
                     state=rng.choice(('early', 'late', 'halos')), chan=chan,
                     cell=0.0 if own else round(rng.uniform(0.7, 2.5), 3),
                     offset=0.0 if own else round(rng.uniform(0.0, 3.0), 3),
                     grad=rng.random() < 0.5)
    grad = rng.random() < 0.5
    ratio = rng.choice((1.0, 2.0))
    if kind == 'force':
        return _case(kind, _grid(rng, 24, 256), ratio=ratio, grad=grad,
                     state=rng.choice(('early', 'mid', 'late')))
    if grad:
        return _case(kind, _grid(rng, 24, 256), ratio=ratio, grad=True, state='mid', da=DA_FINE,
                     steps=rng.randint(2, 6))
    return _case(kind, _grid(rng, 24, 256), ratio=ratio, state=rng.choice(('early', 'mid', 'late')),
                 steps=rng.randint(2, 12))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dims(case):
    return case['g0'], case['g1'], case['g2']


def _a_start(case):
    return STATES[case['state']][0]


def _a_stop(case):
    return _a_start(case) + max(case['steps'], 1) * case['da']


def _conf(case):
    ratio = case['ratio']
    return pm.Configuration(1.0, _dims(case), mesh_shape=int(ratio) if ratio == int(ratio) else ratio,
                            a_start=_a_start(case), a_stop=_a_stop(case), a_nbody_maxstep=case['da'])


def _kvec(shape, spacing=1.0, dtype=torch.float64, device='cuda'):
    ks = [np.fft.fftfreq(n) for n in shape[:-1]] + [np.fft.rfftfreq(shape[-1])]
    out = []
    for i, k in enumerate(ks):
        k = torch.from_numpy(k * (2 * math.pi / spacing)).to(device=device, dtype=dtype)
        out.append(k.reshape((1,) * i + (-1,) + (1,) * (len(ks) - i - 1)))
    return out


def _linear_field(shape, gen):
    """Half spectrum (unnormalised) of a Gaussian field with power ~ k / (1 + (k / k0)^2)^1.5."""
    f = torch.fft.rfftn(torch.randn(shape, generator=gen, device='cuda'))
    k2 = sum(k * k for k in _kvec(shape, dtype=torch.float32))
    k2[0, 0, 0] = 1
    f = f * (k2 ** 0.25 * (1 + k2 * 100) ** -0.75)
    f[0, 0, 0] = 0
    return f, k2


def _zeldovich(shape, gen, rms):
    """Displacements (n, 3) in units of the particle spacing, of this rms per component."""
    f, k2 = _linear_field(shape, gen)
    d = [torch.fft.irfftn(1j * k / k2 * f, s=shape).reshape(-1)
         for k in _kvec(shape, dtype=torch.float32)]
    d = torch.stack(d, dim=1)
    return d * (rms / d.std())


def _particles(case, conf, gen):
    """Particles of the case's state: (pmid, disp, vel)."""
    grid = pm.Particles.gen_grid(conf)
    psi = _zeldovich(_dims(case), gen, STATES[case['state']][1])
    a = _a_start(case)
    vel = psi * (a * a * math.sqrt(OMEGA_M / a ** 3 + 1 - OMEGA_M))
    if case['state'] == 'halos':
        # three of ten particles of each 16^3 Lagrangian block fall onto the block's centre
        shape = _dims(case)
        q = torch.stack(torch.meshgrid(*[torch.arange(n, device='cuda', dtype=torch.float32)
                                         for n in shape], indexing='ij'), -1).reshape(-1, 3)
        take = torch.rand(q.shape[0], generator=gen, device='cuda') < 0.3
        centre = torch.floor(q / 16) * 16 + 8
        fall = centre - q + 0.4 * torch.randn(q.shape, generator=gen, device='cuda')
        psi = torch.where(take[:, None], fall, psi)
    return grid.pmid, (grid.disp + psi).contiguous(), vel.contiguous()


def _target_shape(case, conf):
    """Shape of the mesh that 'scatter' and 'gather' use."""
    if not case['cell']:
        return tuple(conf.mesh_shape)
    return tuple(max(1, int(m / case['cell'])) for m in conf.mesh_shape)


def _mesh_args(case, conf):
    if not case['cell']:
        return {}
    return {'offset': case['offset'] * conf.cell_size, 'cell_size': case['cell'] * conf.cell_size}


def prepare(case, seed):
    gen = torch.Generator(device='cuda')
    gen.manual_seed(1000003 * int(seed) + 17)
    kind, shape = case['kind'], _dims(case)
    s = {'case': case}
    if kind == 'powspec':
        f, _ = _linear_field(shape, gen)
        s['f'] = 1 + torch.fft.irfftn(f, s=shape)
        if case['cross']:
            f, _ = _linear_field(shape, gen)
            s['g'] = 1 + torch.fft.irfftn(f, s=shape)
        return s
    s['conf'] = conf = _conf(case)
    s['cosmo'] = pm.boltzmann(pm.SimpleLCDM(conf), conf, transfer=False, varlin=False)
    n = conf.ptcl_num
    if kind == 'lpt':
        s['modes'] = (30 * _linear_field(shape, gen)[0]).contiguous()
        if case['grad']:
            s['modes'].requires_grad_()
            s['cot'] = [torch.randn((n, 3), generator=gen, device='cuda') for _ in range(2)]
        return s
    pmid, disp, vel = _particles(case, conf, gen)
    if case['grad']:
        disp.requires_grad_()
        vel.requires_grad_()
    s['ptcl'] = pm.Particles(conf, pmid, disp, vel=vel)
    if kind in ('force', 'nbody') and case['grad']:
        # the cotangents of a smooth objective of the positions: displacement-like fields, the
        # velocities' a drift smaller
        s['cot'] = [_zeldovich(shape, gen, r).contiguous()
                    for r in ((1.0,) if kind == 'force' else (1.0, 0.1))]
    if kind in ('scatter', 'gather'):
        chan = (case['chan'],) if case['chan'] else ()
        target = _target_shape(case, conf) + chan
        if kind == 'gather':
            s['mesh'] = torch.randn(target, generator=gen, device='cuda')
            if case['grad']:
                s['mesh'].requires_grad_()
                s['cot'] = [torch.randn((n,) + chan, generator=gen, device='cuda')]
            s['val'] = torch.zeros((n,) + chan, device='cuda')
        else:
            s['mesh'] = torch.zeros(target, device='cuda') if case['cell'] else None
            s['val'] = None
            if chan:
                s['val'] = torch.randn((n,) + chan, generator=gen, device='cuda')
                if case['grad']:
                    s['val'].requires_grad_()
            if case['grad']:
                s['cot'] = [torch.randn(target, generator=gen, device='cuda')]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _with_grads(out, inputs, outputs, cots):
    grads = torch.autograd.grad(outputs, list(inputs.values()), cots)
    res = {k: v.detach() for k, v in out.items()}
    res.update({'grad_' + k: g for k, g in zip(inputs, grads)})
    return res


def run(s):
    case = s['case']
    kind = case['kind']
    if kind == 'powspec':
        k, p, cnt, edges = powspec(s['f'], 1.0, bins=1j / 3 if case['bins'] == 'log' else 1,
                                   g=s.get('g'), deconv=case['deconv'] or None)
        return {'k': k, 'P': p, 'N': cnt, 'edges': edges}
    conf, cosmo = s['conf'], s['cosmo']
    if kind == 'lpt':
        ptcl, _ = pm.lpt(s['modes'], cosmo, conf)
        out = {'pmid': ptcl.pmid, 'disp': ptcl.disp, 'vel': ptcl.vel}
        if not case['grad']:
            return out
        return _with_grads(out, {'modes': s['modes']}, [ptcl.disp, ptcl.vel], s['cot'])
    ptcl = s['ptcl']
    if kind == 'force':
        acc = pm.gravity(_a_start(case), ptcl, cosmo, conf)
        if not case['grad']:
            return {'acc': acc}
        return _with_grads({'acc': acc}, {'disp': ptcl.disp}, [acc], s['cot'])
    if kind == 'nbody':
        end, _ = pm.nbody(ptcl, None, cosmo, conf)
        out = {'disp': end.disp, 'vel': end.vel, 'acc': end.acc}
        if not case['grad']:
            return out
        return _with_grads(out, {'disp': ptcl.disp, 'vel': ptcl.vel}, [end.disp, end.vel], s['cot'])
    if kind == 'scatter':
        mesh = pm.scatter(ptcl, conf, mesh=s['mesh'], val=s['val'], **_mesh_args(case, conf))
        if not case['grad']:
            return {'mesh': mesh}
        ins = {'disp': ptcl.disp}
        if s['val'] is not None:
            ins['val'] = s['val']
        return _with_grads({'mesh': mesh}, ins, [mesh], s['cot'])
    val = pm.gather(ptcl, conf, s['mesh'], val=s['val'], **_mesh_args(case, conf))
    if not case['grad']:
        return {'val': val}
    return _with_grads({'val': val}, {'disp': ptcl.disp, 'mesh': s['mesh']}, [val], s['cot'])


def work(case):
    """Bytes and operations that a pass cannot do without: the particle arrays once per particle
    pass, the meshes once per deposit, gather and axis-split transform (a 3-D transform of a mesh
    takes two passes), and 2.5 log2 of a transform's length per real value."""
    shape = _dims(case)
    n = float(np.prod(shape))
    m = n * case['ratio'] ** 3
    back = 1 if case['grad'] else 0
    fft = 2.5 * m * math.log2(m)
    kind = case['kind']
    if kind == 'powspec':
        k = 2 if case['cross'] else 1
        return {'bytes': k * 8.0 * n, 'flops': k * 2.5 * n * math.log2(n) + 10 * n}
    if kind == 'lpt':
        # modes in, pmid, disp and vel out; six strain and six displacement fields, one source
        b = 4 * n + 30 * n + 4 * (13 * 4 * n)
        return {'bytes': b + back * (28 * n + 4 * (13 * 4 * n)),
                'flops': (1 + back) * (13 * 2.5 * n * math.log2(n) + 60 * n)}
    # one force: density written and read, the half spectrum written and read around the x axis,
    # two spectra written and read, three meshes written and read
    force, force_adj = 60 * m, 56 * m
    if kind == 'force':
        return {'bytes': 18 * n + 30 * n + force + back * (30 * n + 30 * n + force + force_adj),
                'flops': (1 + 3 * back) * 4 * fft + 100 * n}
    if kind == 'nbody':
        steps = case['steps']
        fwd = (steps + 1) * (54 * n + force)
        adj = (steps + 1) * (180 * n + force + force_adj)
        return {'bytes': fwd + back * adj,
                'flops': (steps + 1) * (1 + 2 * back) * (4 * fft + 120 * n)}
    c = max(case['chan'], 1)
    t = (m / case['cell'] ** 3 if case['cell'] else m) * c
    if kind == 'scatter':
        b = 18 * n + 4 * case['chan'] * n + 4 * t
        return {'bytes': b + back * (30 * n + 8 * case['chan'] * n + 4 * t),
                'flops': (1 + back) * n * (30 + 24 * c)}
    return {'bytes': 18 * n + 4 * c * n + 4 * t + back * (30 * n + 4 * c * n + 8 * t),
            'flops': (1 + 2 * back) * n * (30 + 24 * c)}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def _growth_table(a):
    """(3, len(a)) table of D/a and its ln a derivatives of a flat LCDM background at a[i] (a[0] = 0
    stands for deep matter domination), by fourth-order Runge-Kutta in ln a."""
    def rhs(x, y):
        e2 = OMEGA_M * math.exp(-3 * x) + 1 - OMEGA_M
        dlnh = -1.5 * OMEGA_M * math.exp(-3 * x) / e2
        om = 1.5 * OMEGA_M * math.exp(-3 * x) / e2
        return np.array([y[1], -(3 + dlnh - om) * y[0] - (4 + dlnh) * y[1],
                         y[3], om * y[0] ** 2 - (8 + 2 * dlnh - om) * y[2] - (6 + dlnh) * y[3]])

    x = math.log(0.5 * np.finfo(np.float64).eps ** (1 / 3))
    y = np.array([1.0, 0.0, 3 / 7, 0.0])
    rows = [(y, rhs(x, y))]
    for ai in a[1:]:
        end = math.log(ai)
        num = max(16, int(math.ceil((end - x) / 0.01)))
        h = (end - x) / num
        for _ in range(num):
            k1 = rhs(x, y)
            k2 = rhs(x + h / 2, y + h / 2 * k1)
            k3 = rhs(x + h / 2, y + h / 2 * k2)
            k4 = rhs(x + h, y + h * k3)
            y = y + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            x += h
        x = end
        rows.append((y, rhs(x, y)))
    out = []
    for m, i in ((1, 0), (2, 2)):
        g = np.array([r[0][i] for r in rows])
        g1 = np.array([r[0][i + 1] for r in rows])
        g2 = np.array([r[1][i + 1] for r in rows])
        out.append(np.stack([g, m * g + g1, m * m * g + 2 * m * g1 + g2]))
    return out


class _Background:
    """Growth functions as the package defines them: linear interpolation in a of a table at the
    time steps' scale factors."""

    def __init__(self, case):
        a0, a1 = _a_start(case), _a_stop(case)
        nl, nn = math.ceil(a0 * 128), math.ceil((a1 - a0) / case['da'])
        t = np.arange(nn + 1) / nn
        self.a_nbody = a0 * (1 - t) + a1 * t
        self.xa = np.concatenate([np.arange(nl + 1) / nl * a0, self.a_nbody[1:]])
        self.tab = _growth_table(self.xa)

    def growth(self, a, order=1, deriv=0):
        return a ** order * np.interp(a, self.xa, self.tab[order - 1][deriv])

    @staticmethod
    def e2(a):
        return OMEGA_M / a ** 3 + 1 - OMEGA_M

    def g_d(self, a):
        return a ** 2 * math.sqrt(self.e2(a)) * self.growth(a, deriv=1)

    def g_k(self, a):
        dlnh = -1.5 * OMEGA_M / a ** 3 / self.e2(a)
        return a ** 3 * self.e2(a) * (self.growth(a, deriv=2) + (2 + dlnh) * self.growth(a, deriv=1))


class _Cic:
    """Cloud-in-cell neighbours of positions in cells of a mesh: indices and weights."""

    def __init__(self, pos, box, shape):
        # pos in target cells; periodic in `box` target cells; neighbours off `shape` are dropped
        self.pos, self.box, self.shape = pos, box, shape

    def neighbours(self):
        lo = torch.floor(self.pos.detach())
        fr = self.pos - lo
        axes = []
        for a in range(3):
            two = []
            for b in (0, 1):
                i = torch.remainder(lo[:, a] + b, self.box[a])
                w = fr[:, a] if b else 1 - fr[:, a]
                i = torch.floor(i + 1e-9).to(torch.int64)
                w = torch.where(i < self.shape[a], w, torch.zeros_like(w))
                two.append((i.clamp(max=self.shape[a] - 1), w))
            axes.append(two)
        for k in range(8):
            (i, u), (j, v), (m, w) = (axes[a][k >> a & 1] for a in range(3))
            yield (i * self.shape[1] + j) * self.shape[2] + m, u * v * w


def _deposit(cic, val):
    """Mesh (cells, channels) of val (n, channels), or of a number."""
    cells = int(np.prod(cic.shape))
    chan = 1 if not torch.is_tensor(val) else val.shape[1]
    mesh = torch.zeros((cells, chan), dtype=torch.float64, device='cuda')
    for i, w in cic.neighbours():
        mesh = mesh.index_add(0, i, w[:, None] * val)
    return mesh


def _read(cic, mesh):
    out = 0
    for i, w in cic.neighbours():
        out = out + mesh[i] * w[:, None]
    return out


def _chunks(n, size=1 << 24):
    return [slice(i, min(n, i + size)) for i in range(0, n, size)]


def _force64(x, shape, cell, per_ptcl, lean):
    """Accelerations at positions x (n, 3, in cells); `lean`: in pieces and without a graph."""
    parts = _chunks(x.shape[0]) if lean else [slice(None)]
    box = shape
    dens = 0
    for c in parts:
        dens = dens + _deposit(_Cic(x[c], box, shape), per_ptcl)
    kv = _kvec(shape, cell)
    k2 = sum(k * k for k in kv)
    k2[0, 0, 0] = 1
    pot = torch.fft.rfftn(dens.reshape(shape))
    del dens
    pot = pot * (-1.5 * OMEGA_M / k2)
    del k2
    zero = torch.ones_like(pot.real)
    zero[0, 0, 0] = 0
    pot = pot * zero
    del zero
    acc = []
    for k in kv:
        k = torch.where((k.abs() - math.pi / cell).abs() < 1e-6 / cell, torch.zeros_like(k), k)
        mesh = torch.fft.irfftn(-1j * k * pot, s=shape).reshape(-1, 1)
        acc.append(torch.cat([_read(_Cic(x[c], box, shape), mesh) for c in parts]))
    return torch.cat(acc, dim=1)


def _exact_force(case, s, grad):
    conf = s['conf']
    cell, shape = conf.cell_size, tuple(conf.mesh_shape)
    per = conf.mesh_size / conf.ptcl_num
    pmid = s['ptcl'].pmid.double()
    lean = conf.ptcl_num > 1 << 24

    def force(disp):
        return _force64(pmid + disp / cell, shape, cell, per, lean)

    disp = s['ptcl'].disp.detach().double()
    if case['kind'] == 'force':
        disp.requires_grad_(grad)
        acc = force(disp)
        out = {'acc': acc.detach()}
        if case['grad']:
            g = torch.autograd.grad(acc, disp, s['cot'][0].double())[0] if grad else None
            out['grad_disp'] = g
        return out
    vel = s['ptcl'].vel.detach().double()
    disp.requires_grad_(grad)
    vel.requires_grad_(grad)
    bg = _Background(case)
    d, v = disp, vel
    a = bg.a_nbody.tolist()
    acc = force(d)
    f32 = lambda x: float(np.float32(x))  # noqa: E731  (the time-step factors are float32 by definition)
    for a0, a1 in zip(a[:-1], a[1:]):
        h = 0.5 * a0 + 0.5 * a1
        v = v + acc * f32((bg.g_d(h) - bg.g_d(a0)) / bg.g_k(a0))
        d = d + v * f32((bg.growth(a1) - bg.growth(a0)) / bg.g_d(h))
        acc = force(d)
        v = v + acc * f32((bg.g_d(a1) - bg.g_d(h)) / bg.g_k(a1))
    out = {'disp': d.detach(), 'vel': v.detach(), 'acc': acc.detach()}
    if case['grad']:
        gd = gv = None
        if grad:
            gd, gv = torch.autograd.grad([d, v], [disp, vel], [c.double() for c in s['cot']])
        out.update(grad_disp=gd, grad_vel=gv)
    return out


def _exact_mesh(case, s):
    conf = s['conf']
    cell = conf.cell_size * (case['cell'] or 1.0)
    off = conf.cell_size * case['offset'] if case['cell'] else 0.0
    if case['cell']:
        return None   # the wrapped fractions of a foreign mesh are the package's own definition
    shape = _target_shape(case, conf)
    disp = s['ptcl'].disp.detach().double().requires_grad_(case['grad'])
    pos = (s['ptcl'].pmid.double() * conf.cell_size + disp - off) / cell
    cic = _Cic(pos, shape, shape)
    if case['kind'] == 'scatter':
        val = conf.mesh_size / conf.ptcl_num
        if s['val'] is not None:
            val = s['val'].detach().double().requires_grad_(case['grad'])
        mesh = _deposit(cic, val).reshape(shape + ((case['chan'],) if case['chan'] else ()))
        out = {'mesh': mesh.detach()}
        if case['grad']:
            ins = [disp] + ([val] if s['val'] is not None else [])
            g = torch.autograd.grad(mesh, ins, s['cot'][0].double())
            out.update(zip(('grad_disp', 'grad_val'), g))
        return out
    mesh = s['mesh'].detach().double().requires_grad_(case['grad'])
    val = _read(cic, mesh.reshape(-1, case['chan']))
    out = {'val': val.detach()}
    if case['grad']:
        g = torch.autograd.grad(val, [disp, mesh], s['cot'][0].double())
        out.update(zip(('grad_disp', 'grad_mesh'), g))
    return out


def _exact_lpt(case, s):
    conf = s['conf']
    shape = _dims(case)
    modes = s['modes'].detach().to(torch.complex128).requires_grad_(case['grad'])
    kv = _kvec(shape)
    kz = [torch.where((k.abs() - math.pi).abs() < 1e-6, torch.zeros_like(k), k) for k in kv]
    k2 = sum(k * k for k in kv)
    inv = torch.where(k2 > 0, -1 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    pot = [modes * inv]
    phi = {}
    for i in range(3):
        for j in range(i, 3):
            ki, kj = (kv[i], kv[j]) if i == j else (kz[i], kz[j])
            phi[i, j] = torch.fft.irfftn(-ki * kj * pot[0], s=shape)
    src = (phi[0, 0] * phi[1, 1] + phi[0, 0] * phi[2, 2] + phi[1, 1] * phi[2, 2]
           - phi[0, 1] ** 2 - phi[0, 2] ** 2 - phi[1, 2] ** 2)
    pot.append(torch.fft.rfftn(src) * inv)
    bg = _Background(case)
    a = _a_start(case)
    grid = pm.Particles.gen_grid(conf)
    disp, vel = grid.disp.double(), torch.zeros((conf.ptcl_num, 3), dtype=torch.float64, device='cuda')
    for o in (0, 1):
        g = torch.stack([torch.fft.irfftn(-1j * k * pot[o], s=shape).reshape(-1) for k in kz], dim=1)
        disp = disp + bg.growth(a, order=o + 1) * g
        vel = vel + a * a * math.sqrt(bg.e2(a)) * bg.growth(a, order=o + 1, deriv=1) * g
    out = {'pmid': grid.pmid, 'disp': disp.detach(), 'vel': vel.detach()}
    if case['grad']:
        out['grad_modes'] = torch.autograd.grad([disp, vel], modes,
                                                [c.double() for c in s['cot']])[0]
    return out


def _exact_powspec(case, s):
    shape = _dims(case)
    f = torch.fft.rfftn(s['f'].double())
    if case['cross']:
        p = f * torch.fft.rfftn(s['g'].double()).conj()
    else:
        p = f.real ** 2 + f.imag ** 2
    kv = _kvec(shape, 2 * math.pi)   # cycles per cell
    k = torch.sqrt(sum(q * q for q in kv))
    if case['deconv']:
        for q in kv:
            p = p * torch.sinc(q) ** -case['deconv']
    num = torch.full(k.shape, 2.0, dtype=torch.float64, device='cuda')
    num[..., 0] = 1
    if shape[-1] % 2 == 0:
        num[..., -1] = 1
    kf, kmax = 1 / max(shape), 0.5 * math.sqrt(3)
    if case['bins'] == 'log':
        nb = 1 + math.ceil(math.log2(kmax / kf) * 3) + all(n % 2 == 0 for n in shape)
        cut = 1 + math.ceil(math.log2(0.5 / kf) * 3)
        edges = kf * 2 ** (torch.arange(nb, dtype=torch.float64, device='cuda') / 3)
    else:
        nb, cut = 1 + math.ceil(kmax / kf), 1 + math.ceil(0.5 / kf)
        edges = kf * torch.arange(nb, dtype=torch.float64, device='cuda')
    b = torch.bucketize(k, edges, right=case['bins'] == 'log').reshape(-1).clamp(max=nb)

    def binned(x):
        x = x.reshape(-1)
        return torch.zeros(nb + 1, dtype=x.dtype, device='cuda').index_add(0, b, x)[1:cut]

    cnt = binned(num)
    return {'k': binned(k * num) / cnt * 2 * math.pi,
            'P': binned(p * num) / cnt / float(np.prod(shape)),
            'N': cnt, 'edges': edges[:cut] * 2 * math.pi}


def exact(case, seed):
    kind = case['kind']
    if kind == 'nbody' and case['state'] == 'late' and case['steps'] > 8:
        return None   # strongly clustered runs amplify rounding: 64 bits are another trajectory
    s = prepare(case, seed)
    if kind == 'powspec':
        return _exact_powspec(case, s)
    if kind == 'lpt':
        return _exact_lpt(case, s)
    if kind in ('scatter', 'gather'):
        return _exact_mesh(case, s)
    # a graph through every step in 64 bits only where it fits
    n = s['conf'].ptcl_num + 2 * s['conf'].mesh_size
    grad = case['grad'] and n * max(case['steps'], 1) < 1 << 30
    with torch.set_grad_enabled(grad):
        return _exact_force(case, s, grad)
