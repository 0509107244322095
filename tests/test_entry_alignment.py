"""Entry points that read complex values in pairs, or their scratch 16 bytes at a time,
refuse pointers that are not aligned for that before anything is launched: on the device
such a read is a fault.  Runs without a GPU: the addresses are never read."""

import ctypes

import pytest

from pmwd_gb300 import _lib

ALIGN = -3   # PMX_ERR_ALIGN
OK = 0x10000


def _i64(*v):
    return (_lib.c_i64 * len(v))(*v)


GRID, ST = _i64(64, 64, 64), _i64(64 * 33, 33, 1, 64 * 64 * 33)
FAC = (_lib.c_f * 4)(1, 1, 1, 1)
# entry point, its arguments by name in order, the names that have to be aligned, and on how much
ENTRIES = [
    ('pmx_lpt_strain', dict(g=GRID, tab=OK, modes=OK, s=1.0, spec=OK, st=None), ('modes', 'spec'), 8),
    ('pmx_lpt_grad', dict(g=GRID, tab=OK, modes=OK, s=1.0, src2=OK, strides=ST, spec=OK, st=None),
     ('modes', 'src2', 'spec'), 8),
    ('pmx_lpt_src_adj', dict(g=GRID, tab=OK, spec=OK, strides=ST, s=1.0, out=OK, st=None),
     ('spec', 'out'), 8),
    ('pmx_lpt_modes_adj', dict(g=GRID, tab=OK, C=OK, S=OK, strides=ST, s=1.0, out=OK, ost=ST, st=None),
     ('C', 'S', 'out'), 8),
    ('pmx_lpt_solve', dict(g=GRID, tab=OK, modes=OK, s=1.0, orders=2, fac=FAC, scratch=OK, pmid=OK,
                           disp=OK, vel=OK, st=None), ('modes',), 8),
    ('pmx_lpt_solve', dict(g=GRID, tab=OK, modes=OK, s=1.0, orders=2, fac=FAC, scratch=OK, pmid=OK,
                           disp=OK, vel=OK, st=None), ('scratch',), 16),
    ('pmx_powspec_bin_layout', dict(F=OK, G=OK, nb=1, g=GRID, kx=OK, ky=OK, kz=OK, e=OK, ne=4,
                                    right=0, nbin=4, deconv=0.0, k=OK, p=OK, n=OK, hm=0, scratch=OK,
                                    st=None), ('F', 'G', 'scratch'), 8),
]


@pytest.mark.parametrize('name, args, names, to', ENTRIES,
                         ids=[f'{e[0]}-{e[3]}' for e in ENTRIES])
def test_misaligned_pointers_are_refused(name, args, names, to):
    for which in names:
        for off in (4, to // 2, to - 4):
            bad = dict(args, **{which: OK + off})
            conv = [ctypes.c_void_p(v) if isinstance(v, int) and v >= OK else v
                    for v in bad.values()]
            assert getattr(_lib.load(), name)(*conv) == ALIGN, (which, off)
