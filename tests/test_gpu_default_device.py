"""powspec under a default device: bin edges are then made on the GPU."""

import pytest
import torch

from pmwd_gb300.spec_util import powspec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape', [(16, 32, 8), (9, 12, 10)])
@pytest.mark.parametrize('bins', [1j / 3, 2, (0, 0.1, 0.3, 0.5)])
def test_powspec_under_a_default_device(cuda, shape, bins):
    f = torch.randn(shape, device=cuda)
    want = powspec(f, 1.3, bins=bins, deconv=2)
    for _ in range(2):
        with torch.device(cuda):
            got = powspec(f, 1.3, bins=bins, deconv=2)
        for a, b in zip(got, want):
            assert a.device == b.device
            # float64 sums in another order (P of float32 products); empty bins are 0 / 0
            torch.testing.assert_close(a, b, rtol=1e-9, atol=0, equal_nan=True)
