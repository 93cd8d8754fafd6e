"""hermes_field_sum and hermes_field_shift at the edges of their vector loads
and block shares, aligned and not.

Sum: 15 float32 two-sum steps lose at most 15 * 2^-47 of the group's sum of
|x| (the error terms are added in float32) and the float64 additions at most
n / 16 * 2^-53 of the total: 1e-12 of sum |x| covers n up to 2^21.  Shift: one
rounding of x - r plus the rounding of its error term, at most one unit in
the last place from the correctly rounded value."""
import math

import numpy as np
import pytest
import torch

from pyhermes_gb300 import kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4096, 16385, 1 << 21])
@pytest.mark.parametrize("off", [0, 1])
def test_field_sum(n, off):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = (torch.randn(n + 1, generator=g, device="cuda") * torch.exp(3 * torch.randn(n + 1, generator=g, device="cuda")))[off:off + n]
    h = x.cpu().numpy().astype(np.float64)
    assert abs(kernels.field_sum(x) - math.fsum(h)) <= 1e-12 * np.abs(h).sum()


@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 16385])
@pytest.mark.parametrize("off", [0, 1])
def test_field_shift(n, off):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.exp(4 * torch.randn(n + 1, generator=g, device="cuda"))[off:off + n]
    for r in (0.0, 1.0 / 3.0, float(x[0].item()), 1e-9, 5e4):
        ref = (x.double() - r).float().cpu().numpy()
        got = kernels.field_shift(x, r).cpu().numpy()
        assert np.all(np.abs(got - ref) <= np.spacing(np.abs(ref))), r


def test_special_values():
    x = torch.tensor([float("inf"), 1.0, float("-inf"), float("nan"), 2.0], device="cuda")
    y = kernels.field_shift(x, 0.5).cpu().numpy()
    np.testing.assert_array_equal(y, [np.inf, 0.5, -np.inf, np.nan, 1.5])
    assert not math.isfinite(kernels.field_sum(torch.full((4096,), float("inf"), device="cuda")))
    assert kernels.field_sum(torch.zeros(0, device="cuda")) == 0.0
