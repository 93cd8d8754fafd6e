"""Pair products where large modes of one kernel value cancel: what they leave
is not lost in the sums over the modes that share it.  The kernel value is a
dozen float32 roundings: 2e-6 of it."""
import numpy as np
import pytest
import torch

from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.window import WindowFunc, pair_products

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()
J, L = 4, 16
INFO = {"J": J, "box_size": 16.0, "phi_resolution": 1024, "wavelet_mode": "db2", "wavelet_level": 10, "phi_array": PHI}
RADIAL = ({"type": "gdw", "len_args": {"R": 1.0}}, {"type": "gaussian", "len_args": {"R": 0.5}}, {"type": "laplacian"})
CYL = ({"type": "ring", "len_args": {"R": 0.4, "H": 0.3}}, {"type": "cylinder", "len_args": {"R": 0.5, "H": 0.4}})


@pytest.mark.parametrize("where,kinds", [("columns", RADIAL), ("columns", CYL), ("places", RADIAL)])
def test_cancelling_modes(where, kinds):
    """T = 2^24, 1, -2^24: the sum is 1, which float32 additions in the order
    of the modes would lose."""
    s = [torch.zeros((L, L, L // 2 + 1), dtype=torch.complex64, device="cuda") for _ in range(2)]
    at = {"columns": [(2, 1, 3), (L - 2, 1, 3), (2, L - 1, 3)], "places": [(5, 3, 2), (5, 2, 3), (3, 2, 5)]}[where]
    for m, a, b in zip(at, (4096.0, 1.0, 4096.0), (4096.0, 1.0, -4096.0)):
        s[0][m], s[1][m] = a, b
    wins = [WindowFunc(p, INFO, device="cuda") for p in kinds]
    got, _ = pair_products(s, [(0, 1)], wins)
    for k, w in enumerate(wins):
        want = 2.0 * float(np.asarray(w.as_array())[at[1]]) / float(L) ** 6
        assert want != 0.0 and abs(got[k, 0] - want) <= 2e-6 * abs(want), (k, got[k, 0], want)


def test_products_near_the_largest_float32():
    """Three places of |T| = 2^126.6: their sum is above float32's range, the
    result is not."""
    s = [torch.zeros((L, L, L // 2 + 1), dtype=torch.complex64, device="cuda")]
    for m in [(5, 3, 2), (5, 2, 3), (3, 2, 5)]:
        s[0][m] = 2.0 ** 62.8
    wins = [WindowFunc(p, INFO, device="cuda") for p in RADIAL]
    got, _ = pair_products(s, [(0, 0)], wins)
    for k, w in enumerate(wins):
        want = 3 * 2.0 * (float(np.float32(2.0 ** 62.8)) ** 2) * float(np.asarray(w.as_array())[5, 3, 2]) / float(L) ** 6
        assert abs(got[k, 0] - want) <= 2e-6 * abs(want), (k, got[k, 0], want)
