"""Float64 host arithmetic for calls that need no gradient.

The initial-condition path evaluates a few hundred scalars per call: the
linear power spectrum on the table of distinct |k| (modes.py:67-117 via
boltzmann.py:399-455) and the growth factors at a_start (lpt.py:197-210); an
N-body run the drift and kick factors of its steps (nbody.py:12-36).
As torch CPU tensors these are ~10^2 dispatched ops (one to three milliseconds);
when nothing needs a gradient they are evaluated here in NumPy with the
same formulas and the same order of operations as the torch code in
``boltzmann`` and ``cosmology``, so both give the same float32 results.
"""

import math

import numpy as np
import torch


def _f(x):
    return float(x.detach()) if torch.is_tensor(x) else float(x)


def interp(x, xp, fp):
    """boltzmann.interp (``jnp.interp``, clamped) on NumPy float64 arrays."""
    x = np.asarray(x, np.float64)
    n = xp.shape[0]
    i = np.clip(np.searchsorted(xp, x, side='right'), 1, n - 1)
    df = fp[i] - fp[i - 1]
    dx = xp[i] - xp[i - 1]
    delta = x - xp[i - 1]
    f = np.where(dx == 0, fp[i], fp[i - 1] + (delta / np.where(dx == 0, 1, dx)) * df)
    f = np.where(x < xp[0], fp[0], f)
    return np.where(x > xp[-1], fp[-1], f)


def needs_grad(*objs):
    """Whether autograd has to see any tensor of these objects (tensors,
    or dataclasses such as Cosmology holding tensors)."""
    if not torch.is_grad_enabled():
        return False
    for o in objs:
        if torch.is_tensor(o):
            if o.requires_grad:
                return True
        elif hasattr(o, '__dict__'):
            if any(torch.is_tensor(v) and v.requires_grad for v in vars(o).values()):
                return True
    return False


def growth(a, cosmo, conf, order=1, deriv=0, tables=None):
    """boltzmann.growth at a scalar a; tables = (conf.growth_a, cosmo.growth)
    as NumPy arrays when the caller already has them."""
    xp, tab = tables if tables is not None else (conf.growth_a.numpy(),
                                                 cosmo.growth.detach().cpu().numpy())
    return a ** order * float(interp(a, xp, tab[order - 1][deriv]))


def E2(a, cosmo):
    """cosmology.E2 at a scalar a."""
    Om, Ok, w0, wa = (_f(cosmo.Omega_m), _f(cosmo.Omega_k), _f(cosmo.w_0), _f(cosmo.w_a))
    Ode = 1 - (Om + Ok)
    de_a = a ** (-3 * (1 + w0 + wa)) * math.exp(-3 * wa * (1 - a))
    return Om * a ** -3 + Ok * a ** -2 + Ode * de_a


class _Background:
    """The growth factors of nbody.py:12-22 at an array of scale factors; the
    interpolation's intervals and the expansion rate are worked out once."""

    def __init__(self, a, xp, tab, cosmo):
        self.a, self.tab = a, tab[0]
        self.i = np.clip(np.searchsorted(xp, a, side='right'), 1, len(xp) - 1)
        lo = xp[self.i - 1]
        dx = xp[self.i] - lo
        self.r = (a - lo) / np.where(dx == 0, 1, dx)
        self.flat = dx == 0
        self.below, self.above = a < xp[0], a > xp[-1]
        self.edges = bool((self.flat | self.below | self.above).any())
        self.Om, self.Ok = _f(cosmo.Omega_m), _f(cosmo.Omega_k)
        self.Ode = 1 - (self.Om + self.Ok)
        w0, wa = _f(cosmo.w_0), _f(cosmo.w_a)
        self.p, self.q = -3 * (1 + w0 + wa), -3 * wa
        self.de_a = a ** self.p * np.exp(self.q * (1 - a))
        self.E2 = self.Om * a ** -3 + self.Ok * a ** -2 + self.Ode * self.de_a

    def growth(self, deriv=0):
        fp = self.tab[deriv]
        hi, lo = fp[self.i], fp[self.i - 1]
        f = lo + self.r * (hi - lo)
        if self.edges:   # as interp
            f = np.where(self.flat, hi, f)
            f = np.where(self.below, fp[0], f)
            f = np.where(self.above, fp[-1], f)
        return self.a * f

    def G_D(self):
        return self.a ** 2 * np.sqrt(self.E2) * self.growth(1)

    def G_K(self):
        a = self.a
        H_deriv = 0.5 * (-3 * self.Om * a ** -3 - 2 * self.Ok * a ** -2
                         + self.Ode * self.de_a * (self.p - self.q * a)) / self.E2
        return a ** 3 * self.E2 * (self.growth(2) + (2 + H_deriv) * self.growth(1))


def op_factors(ops, cosmo, conf):
    """nbody.op_factors as a float64 NumPy array: the drift_factor or
    kick_factor (nbody.py:25-36) of every drift and kick, in op order."""
    if cosmo.growth is None:
        raise ValueError('Growth table is empty. Call growth_integ or boltzmann first.')
    xp = np.concatenate((conf.a_lpt.numpy(), conf.a_nbody.numpy()[1:]))   # conf.growth_a
    tab = cosmo.growth.detach().cpu().numpy()
    ops = [o for o in ops if len(o) == 4]
    kick = np.array([o[0].startswith('kick') for o in ops], dtype=bool)
    args = np.array([o[1:] for o in ops], dtype=np.float64).reshape(-1, 3)
    num = int(kick.sum())
    out = np.empty(len(kick))
    k, d = args[kick], args[~kick]
    # kicks: the velocities' G_D at both ends, over G_K of the accelerations
    GD = _Background(np.concatenate((k[:, 2], k[:, 1], d[:, 0])), xp, tab, cosmo).G_D()
    out[kick] = (GD[:num] - GD[num:2 * num]) / _Background(k[:, 0], xp, tab, cosmo).G_K()
    D = _Background(np.concatenate((d[:, 2], d[:, 1])), xp, tab, cosmo).growth()
    out[~kick] = (D[:len(d)] - D[len(d):]) / GD[2 * num:]
    return out


def lpt_factors(cosmo, conf):
    """(lpt_order, 2) float32 array of (D_m, a^2 H dD_m/dlna) at a_start."""
    a = conf.a_start
    xp = np.concatenate((conf.a_lpt.numpy(), conf.a_nbody.numpy()[1:]))   # conf.growth_a
    tab = cosmo.growth.detach().cpu().numpy()
    a2H = a ** 2 * math.sqrt(E2(a, cosmo))
    i = min(max(int(np.searchsorted(xp, a, side='right')), 1), len(xp) - 1)
    rows = []
    for order in range(1, 1 + conf.lpt_order):
        D, dD = (a ** order * float(interp(a, xp[i - 1:i + 1], tab[order - 1][deriv][i - 1:i + 1]))
                 for deriv in (0, 1))
        rows.append((D, a2H * dD))
    return np.asarray(rows, np.float64).astype(np.float32)


def mode_amplitude(k, a, cosmo, conf):
    """sqrt(V P_lin(k)) in float32 (modes.py:102-112 with
    boltzmann.linear_power) at float64 wavenumbers k."""
    T = interp(k, conf.transfer_k.numpy(), cosmo.transfer.detach().cpu().numpy())
    kp = _f(cosmo.k_pivot)
    x = k / kp
    pos = x > 0
    pw = np.where(pos, np.power(np.where(pos, x, 1.0), _f(cosmo.n_s)), 0.0)
    Plin = (0.32 * _f(cosmo.A_s) * kp * pw
            * (math.pi * (conf.c / conf.H_0) ** 2 / _f(cosmo.Omega_m) * T) ** 2)
    if a is not None:
        Plin = Plin * growth(a, cosmo, conf) ** 2
    P32 = Plin.astype(np.float32)
    return np.sqrt(P32 * np.float32(conf.box_vol))
