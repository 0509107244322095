"""Step factors of runs without cosmology gradients (NumPy) against the torch functions that
carry the gradients: the same float32 values for every operation."""

import numpy as np
import pytest


@pytest.mark.parametrize('cosmo_kw', [{}, {'Omega_k_': 0.05, 'w_0_': -0.9, 'w_a_': 0.1}])
@pytest.mark.parametrize('splits', [((0, 0.5), (1, 0.5)), ((0.5, 0), (0.5, 1)),
                                    ((0.5, 0.5), (0.5, 0.5))])
@pytest.mark.parametrize('reverse', [False, True])
@pytest.mark.parametrize('steps', [1, 2, 63])
def test_op_factors(cosmo_kw, splits, reverse, steps):
    import importlib

    import pmwd_gb300 as pg
    from pmwd_gb300 import _hostmath
    nb = importlib.import_module('pmwd_gb300.nbody')
    conf = pg.Configuration(1.0, (8,) * 3, symp_splits=splits, a_nbody_maxstep=1 / steps)
    cosmo = pg.boltzmann(pg.SimpleLCDM(conf, **cosmo_kw), conf, varlin=False)
    for ops in (nb.forward_ops(conf, reverse), nb.adjoint_ops(conf, reverse)):
        want = nb.op_factors(ops, cosmo, conf).numpy()
        got = _hostmath.op_factors(ops, cosmo, conf)
        # float64 powers of two libraries may differ in the last bits
        assert np.allclose(got, want, rtol=1e-12, atol=0)
        assert np.array_equal(got.astype(np.float32), want.astype(np.float32))


def test_op_factors_needs_the_growth_table():
    import importlib

    import pmwd_gb300 as pg
    from pmwd_gb300 import _hostmath
    nb = importlib.import_module('pmwd_gb300.nbody')
    conf = pg.Configuration(1.0, (8,) * 3, a_nbody_maxstep=1 / 2)
    with pytest.raises(ValueError, match='Growth table is empty'):
        _hostmath.op_factors(nb.forward_ops(conf), pg.SimpleLCDM(conf), conf)
