"""pmx_powspec_bin and pmx_powspec_bin_zmajor, which bring their own scratch, against
pmx_powspec_bin_layout with the caller's: same sums, on a power-of-two grid and another."""

import pytest
import torch

from pmwd_gb300 import _lib
from pmwd_gb300 import spec_util as su

pytestmark = pytest.mark.gpu


def _bin(name, F, G, grid, edges, right, deconv, *extra):
    tabs = su._to_device(F.device, *su.fftfreq(grid, None, dtype=torch.float64), edges)
    n = len(edges)
    k, num = (torch.zeros(n, dtype=torch.float64, device=F.device) for _ in range(2))
    p = torch.zeros(n, 2, dtype=torch.float64, device=F.device)
    _lib.call(name, torch.view_as_real(F), None if G is None else torch.view_as_real(G),
              F.shape[0], (_lib.c_i64 * 3)(*grid), *tabs, n, int(right), n, deconv, k, p, num, *extra,
              _lib.stream_ptr(F.device))
    return k, p, num


@pytest.mark.parametrize('grid', [(32, 64, 16), (12, 9, 10)])
@pytest.mark.parametrize('cross', [False, True])
def test_entries_with_own_scratch(cuda, grid, cross):
    gen = torch.Generator(device=cuda).manual_seed(3)
    F, G = (torch.fft.rfftn(torch.randn((2,) + grid, generator=gen, device=cuda), dim=(1, 2, 3))
            .contiguous() for _ in range(2))
    G = G if cross else None
    _, _, edges, right = su._getbins(grid, 1j / 3, True)
    for deconv in (0.0, 2.0):
        for zmajor in (False, True):
            if zmajor and not su._pow2_grid(grid):
                continue   # what pmx_powspec_bin_zmajor takes
            f, g = (x if x is None or not zmajor else x.movedim(-1, -3).contiguous() for x in (F, G))
            nbytes = _lib.load().pmx_powspec_scratch_bytes((_lib.c_i64 * 3)(*grid), len(edges),
                                                           len(edges), int(deconv != 0), 1, int(zmajor))
            scratch = torch.empty(nbytes, dtype=torch.uint8, device=cuda)
            want = _bin('pmx_powspec_bin_layout', f, g, grid, edges, right, deconv, int(zmajor), scratch)
            got = _bin('pmx_powspec_bin_zmajor' if zmajor else 'pmx_powspec_bin', f, g, grid, edges,
                       right, deconv)
            assert torch.equal(got[2], want[2])
            for a, b in zip(got[:2], want[:2]):
                # the same terms, at most 2^15 of them, summed to 2^-46 in any order
                torch.testing.assert_close(a, b, rtol=0, atol=1e-9 * float(b.abs().max()))
