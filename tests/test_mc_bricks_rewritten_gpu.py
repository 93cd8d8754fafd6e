"""The Monte Carlo sums read the field as it is at the call, also when a native
call has rewritten its buffer, which torch's version counter does not see."""
import numpy as np
import pytest
import torch

from pyhermes_gb300 import kernels, mc3pcf
from pyhermes_gb300.phi import sample_scaling_function

pytestmark = pytest.mark.gpu


def test_a_field_rewritten_by_a_deposit():
    J, L, n = 5, 32, 20000
    phi = torch.as_tensor(sample_scaling_function(), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    w = torch.ones(n, dtype=torch.float64, device="cuda")
    cen = torch.rand((3000, 3), generator=g, device="cuda", dtype=torch.float64) * L
    off = mc3pcf.rotation_offsets(4.0, 7.0, 0.2, 5, rng=np.random.RandomState(1))
    eps = torch.zeros((L, L, L), device="cuda")
    seen = []
    # enough triplets and samples for the brick copies
    assert mc3pcf.choose_bricks((eps, eps, eps), J, 3000 * 5) is not False
    for k in range(3):
        pos = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * (1000.0 / (1 + k))
        kernels.deposit(pos, w, J, 1000.0, phi, out=eps)
        want, _ = mc3pcf.triplet_sum(eps, eps, eps, J, cen, off, phi, bricks=False)
        got, _ = mc3pcf.triplet_sum(eps, eps, eps, J, cen, off, phi)
        assert got == want, k
        sample = (eps, eps, eps, J, cen, phi, 4.0, 7.0, 0.2, 20000)
        a = mc3pcf.mc_sample(*sample, seed=k, bricks=False)
        assert a == mc3pcf.mc_sample(*sample, seed=k) == \
            mc3pcf.mc_sample(*sample, seed=k, bricks=mc3pcf.brick_fields(sample[:3], J))
        b = mc3pcf.field_bricks(eps, J)
        assert torch.equal(b, eps.view(L // 2, 2, L // 2, 2, L // 2, 2).permute(0, 2, 4, 1, 3, 5).reshape(-1))
        seen.append(got)
    assert len(set(seen)) == 3


@pytest.mark.parametrize("J", [2, 3, 6])
def test_bricks_at_any_alignment(J):
    """hermes_field_to_bricks by whole bricks and, where the field or the copy
    is not aligned for that, cell by cell."""
    L = 1 << J
    base = torch.rand(L ** 3 + 2, generator=torch.Generator(device="cuda").manual_seed(J), device="cuda")
    for a in (0, 1, 2):
        f = base[a:a + L ** 3]
        want = f.view(L // 2, 2, L // 2, 2, L // 2, 2).permute(0, 2, 4, 1, 3, 5).reshape(-1)
        for b in (0, 1, 4):
            out = torch.zeros(L ** 3 + 4, device="cuda")[b:b + L ** 3]
            assert torch.equal(mc3pcf._to_bricks(f, J, out), want), (a, b)


def test_rule_for_the_copies():
    """The two layouts give the same sums on both sides of the line, and what
    bricks refuse is refused on both."""
    J, L = 6, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    f = [torch.rand((L, L, L), generator=g, device="cuda") for _ in range(3)]
    phi = torch.as_tensor(sample_scaling_function(), device="cuda")
    off = mc3pcf.rotation_offsets(4.0, 7.0, 0.2, 3, rng=np.random.RandomState(1))
    line = 3 * L ** 3 // 128
    assert mc3pcf.choose_bricks(f, J, line - 1) is False and mc3pcf.choose_bricks(f, J, line) is not False
    assert mc3pcf.choose_bricks([None, f[0], f[0]], J, L ** 3 // 128)[0] is None
    for n in (line // 3 - 1, line // 3 + 1):
        c = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * L
        got = [mc3pcf.triplet_sum(*f, J, c, off, phi, samples=True, bricks=b) for b in (True, False, 1, 0, None)]
        assert all(t == got[0][0] and torch.equal(v, got[0][1]) for t, v in got[1:])
        for bad in (f[0].double(), f[0].transpose(0, 1), f[0][1:]):
            with pytest.raises(ValueError):
                mc3pcf.triplet_sum(f[0], f[1], bad, J, c, off, phi)
