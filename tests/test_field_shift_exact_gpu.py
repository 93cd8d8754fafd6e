"""hermes_field_shift gives the bits of the float64 expression (x - r).float():
values at, beside and far from r, ties, subnormals, infinities."""
import numpy as np
import pytest
import torch

from pyhermes_gb300 import kernels

pytestmark = pytest.mark.gpu


def _equal(x, r):
    want = (x.double() - r).float()
    got = kernels.field_shift(x, r)
    same = (got.view(torch.int32) == want.view(torch.int32)) | (got.isnan() & want.isnan())
    assert bool(same.all()), (r, x[~same][:4], got[~same][:4], want[~same][:4])


def test_values_beside_the_mean():
    """x within a few units in the last place of r: the digits of r beyond two
    float32 values decide the rounding."""
    rng = np.random.default_rng(1)
    for r in np.concatenate([rng.uniform(0.5, 2.0, 200) * 10.0 ** rng.integers(-9, 9, 200), -rng.uniform(1.0, 2.0, 20)]):
        rh = np.float32(r)
        k = np.arange(-40, 41)
        _equal(torch.as_tensor((rh + k * np.spacing(np.abs(rh))).astype(np.float32), device="cuda"), float(r))


@pytest.mark.parametrize("off", [0, 1])
def test_values_of_every_size(off):
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((1 << 22) + 2, generator=g, device="cuda") * torch.exp2(
        torch.randint(-40, 40, ((1 << 22) + 2,), generator=g, device="cuda").float())
    x = x[off:off + (1 << 22) + 1]
    for r in (1.0 / 3.0, -7.25e-3, 2.0 ** -24 + 2.0 ** -48, 1.0 + 2.0 ** -24, 1e-30, 3.1e7, 0.0):
        _equal(x, r)


def test_ties_and_special_values():
    x = torch.tensor([0.0, -0.0, 1.0, 2.0, 3.0, 1.0 + 2.0 ** -23, 2.0 ** -126, 2.0 ** -149, -2.0 ** -140, 3.4e38, -3.4e38,
                      float("inf"), float("-inf"), float("nan"), 16777216.0, 16777217.0], device="cuda")
    for r in (0.5, 2.0 ** -24, 2.0 ** -25, 3 * 2.0 ** -25, -2.0 ** -24, 2.0 ** -53, 2.0 ** -150, 2.0 ** -149, 1e-45, 1e300, -1e300,
              3.4028235677973366e38, 0.0, float("inf"), float("nan")):
        _equal(x, r)
