"""The two-word accumulation in float32 roundings: the float64 field is the
int64 sums times a power of two, so it equals them bit for bit.  Particle
counts from which the hi parts fit, on both sides of the numbers of records a
tile may hold for split bits 21 and 20 (682, 1365) and of the whole path; weights
of both signs, contributions below one quantum and ties of the rounding."""
import numpy as np
import pytest
import torch

from pyhermes_gb300 import kernels
from pyhermes_gb300.phi import sample_scaling_function
from test_deposit_exact_gpu import _exact_deposit

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()


@pytest.mark.parametrize("J,n,scatter", [(5, 600_000, 1.0), (7, 540_000, 1.0), (7, 900_000, 1.0), (7, 1_500_000, 0.6),
                                         (8, 1_000_000, 0.02)])
def test_words_hold_the_int64_sums(J, n, scatter):
    rng = np.random.default_rng(n + J)
    box = 1000.0
    pos = rng.uniform(0.0, box, (n, 3))
    k = int(n * (1.0 - scatter))
    pos[:k] = np.mod(rng.normal(300.0, 120.0, (k, 3)), box)
    w = rng.uniform(-1.0, 1.5, n)
    w[::3] = np.exp2(-rng.integers(0, 60, w[::3].size))
    w[1::3] = np.round(w[1::3] * 8) / 8
    t = lambda a: torch.as_tensor(a, device="cuda")
    eps, _, _ = kernels.deposit(t(pos), t(w), J, box, t(PHI), out_dtype=torch.float64)
    assert np.array_equal(eps.cpu().numpy().reshape(-1), _exact_deposit(pos, w, J, box))
