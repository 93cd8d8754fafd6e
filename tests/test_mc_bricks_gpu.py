"""The whole-brick gather against the C-order one: the same sums in the same
order, so the same bits, at cell and brick edges, across the periodic wrap
and below zero, from the smallest grid up; a NaN reaches exactly the stencils
that hold its cell; rotations shared by several threads give the sum of the
per-triplet products (float32 partial sums of at most n_rot terms: n_rot 2^-24
of the sum of |f|)."""
import numpy as np
import pytest
import torch

from pyhermes_gb300 import mc3pcf
from pyhermes_gb300.phi import sample_scaling_function

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()


def _case(J, nc, n_rot):
    L = 1 << J
    rng = np.random.default_rng(J)
    c = rng.uniform(0.0, L, (nc, 3))
    c[:8] = [[0, 0, 0], [L - 1, L - 1, L - 1], [1, 2, 3 % L], [0.5, L - 0.25, 2], [2 ** -40, 1 - 2 ** -40, L - 2 ** -30],
             [L / 2, L / 2 - 1e-12, 1], [3 % L, 0, L - 1e-9], [1.0 / 1024, 2 + 1023.0 / 1024, 0.75]]
    off = rng.normal(0.0, L / 3, (n_rot, 6))
    off[0] = 0.0
    off[1] = [-L, -1, -0.5, 1, L, -2 ** -45]
    g = torch.Generator(device="cuda").manual_seed(J)
    f = [torch.randn((L,) * 3, generator=g, device="cuda") for _ in range(3)]
    return f, torch.as_tensor(c, device="cuda"), off, torch.as_tensor(PHI, device="cuda")


@pytest.mark.parametrize("J", [2, 3, 6, 9])
def test_bricks_give_the_same_bits(J):
    f, c, off, phi = _case(J, 500, 7)
    f[1][1, 2, 3] = float("nan")
    a, sa = mc3pcf.triplet_sum(*f, J, c, off, phi, samples=True, bricks=False)
    b, sb = mc3pcf.triplet_sum(*f, J, c, off, phi, samples=True, bricks=True)
    assert np.array_equal(sa.cpu().numpy(), sb.cpu().numpy(), equal_nan=True)
    assert bool(torch.isnan(sa).any()) and not bool(torch.isnan(sa).all())
    # fields that are not 32-byte (bricks) or 16-byte (C order) aligned are read cell by cell
    off1 = torch.empty(8 ** J + 1, device="cuda")[1:].view_as(f[2]).copy_(f[2])
    _, sc = mc3pcf.triplet_sum(f[0], f[1], off1, J, c, off, phi, samples=True, bricks=True)
    assert np.array_equal(sb.cpu().numpy(), sc.cpu().numpy(), equal_nan=True)
    _, sd = mc3pcf.triplet_sum(f[0], f[1], off1, J, c, off, phi, samples=True, bricks=False)
    assert np.array_equal(sb.cpu().numpy(), sd.cpu().numpy(), equal_nan=True)
    p = mc3pcf.interp(f[2], J, c, phi)
    assert torch.equal(p, mc3pcf.interp(off1, J, c, phi))


@pytest.mark.parametrize("nc,n_rot", [(8, 1), (8, 15), (9, 64), (300, 100), (5000, 17)])
def test_shared_rotations(nc, n_rot):
    f, c, off, phi = _case(5, max(nc, 8), max(n_rot, 2))
    c, off = c[:nc], off[:n_rot]
    total, _ = mc3pcf.triplet_sum(*f, 5, c, off, phi)
    _, s = mc3pcf.triplet_sum(*f, 5, c, off, phi, samples=True)
    s = s.double().cpu().numpy()
    assert abs(total - s.sum()) <= n_rot * 2.0 ** -24 * np.abs(s).sum()


def test_morton_order_matches_host():
    g = torch.Generator(device="cuda").manual_seed(1)
    c = torch.rand((3000, 3), generator=g, device="cuda", dtype=torch.float64) * 700 - 90
    keys = mc3pcf.morton_order(c.cpu(), 512)
    cells = torch.floor(c).long() & 511
    # the same cells in the same order (equal cells may swap)
    assert torch.equal(cells[mc3pcf.morton_order(c, 512)].cpu(), cells.cpu()[keys])
