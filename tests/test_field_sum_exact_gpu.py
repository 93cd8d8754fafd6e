"""hermes_field_sum at sizes where a thread adds several loads of float4 at a
time in float32: as close as float64 additions, and with their infinities.

Sixteen values of one thread, every other value zero: the float32 sums with
their errors carry them to far below 2^-53 of the sum of |x|, of which the two
float64 additions that end the group lose at most 2^-53 each: 4 2^-53 of it."""
import math

import numpy as np
import pytest
import torch

from pyhermes_gb300 import kernels

pytestmark = pytest.mark.gpu


def _stride():
    # float4 values between a thread's loads
    return torch.cuda.get_device_properties(0).multi_processor_count * 8 * 256


def test_a_group_of_wide_range():
    st = _stride()
    rng = np.random.default_rng(2)
    x = torch.zeros(16 * st, dtype=torch.float32, device="cuda")
    worst = 0.0
    for _ in range(64):
        h = (rng.standard_normal(16) * 2.0 ** rng.uniform(-30, 0, 16)).astype(np.float32)
        t = int(rng.integers(st))
        x.zero_()
        for k in range(4):
            x[4 * (t + k * st):4 * (t + k * st) + 4] = torch.as_tensor(h[4 * k:4 * k + 4], device="cuda")
        d = h.astype(np.float64)
        worst = max(worst, abs(kernels.field_sum(x) - math.fsum(d)) / np.abs(d).sum())
    assert worst <= 4 * 2.0 ** -53


@pytest.mark.parametrize("off", [0, 1])
def test_infinities_and_float32_overflow(off):
    n = 16 * _stride() + 5
    x = torch.full((n + 1,), 3e38, dtype=torch.float32, device="cuda")[off:off + n]
    assert abs(kernels.field_sum(x) / (n * float(np.float32(3e38))) - 1.0) < 1e-12
    x[7] = float("inf")
    assert kernels.field_sum(x) == math.inf
    x[7] = float("-inf")
    assert kernels.field_sum(x) == -math.inf
    x[9] = float("inf")
    assert math.isnan(kernels.field_sum(x))
    x[7] = 0.0
    x[9] = float("nan")
    assert math.isnan(kernels.field_sum(x))
