"""Pair products of isotropic bins by the histogram over |k|^2 of the folded
spectrum, against the generic per-mode kernel on the same bins.  All five
isotropic windows, one to four spectrum pairs (shared and distinct spectra),
with and without the k = 0 mode, from the smallest grid up.

Both passes form products of float32 spectra, weights and window values (each
product off by a few 2^-24) and add them in float64, in different orders and
groupings of at most 8 float32 terms: 1e-6 of the sum of |T K|, which the
bins' largest |value| at R = 0 (W = 1) is for an auto pair.  The bound is
taken against that value."""
import numpy as np
import pytest
import torch

from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.window import WindowFunc, pair_products, rfft_field

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()
KINDS = ({"type": "shell", "len_args": {"R": 0.0}}, {"type": "sphere", "len_args": {"R": 70.0}},
         {"type": "gaussian", "len_args": {"R": 25.0}}, {"type": "shell", "len_args": {"R": 130.0}},
         {"type": "thick_shell", "len_args": {"R": 90.0, "delta_R": 15.0}},
         {"type": "gaussian_shell", "len_args": {"R_shell": 60.0, "R_smooth": 12.0}})


def _win(J, p, bandwidth=1):
    info = {"J": J, "box_size": 1000.0, "phi_resolution": 1024, "wavelet_mode": "db2", "wavelet_level": 10,
            "phi_array": PHI}
    return WindowFunc(p, info, bandwidth=bandwidth, device="cuda")


@pytest.mark.parametrize("J,n_pairs,exclude_k0,mode", [(2, 1, False, "octant"), (3, 4, True, "octant"),
                                                       (5, 2, False, "full_rfft"), (6, 3, True, "octant"),
                                                       (7, 4, False, "octant"), (7, 1, True, "full_rfft")])
def test_radial_histogram_matches_generic_kernel(J, n_pairs, exclude_k0, mode):
    L = 1 << J
    g = torch.Generator(device="cuda").manual_seed(J * 10 + n_pairs)
    fields = [torch.exp(torch.randn((L, L, L), generator=g, device="cuda")) for _ in range(3)]
    spectra = [rfft_field(f) for f in fields]
    pairs = [(0, 0), (0, 1), (2, 1), (2, 2)][:n_pairs]
    bins = [_win(J, dict(p, kernel_mode=mode)) for p in KINDS]
    hist, k0h = pair_products(spectra, pairs, bins, exclude_k0=exclude_k0)
    # one window of another family sends every bin through the generic kernel
    extra = _win(J, {"type": "cubic", "len_args": {"Lx": 30.0, "Ly": 20.0, "Lz": 10.0}})
    gen, k0g = pair_products(spectra, pairs, bins + [extra], exclude_k0=exclude_k0)
    auto, _ = pair_products(spectra, [(0, 0), (1, 1), (2, 2)], bins[:1] + [extra], exclude_k0=exclude_k0)
    size = {p: np.sqrt(auto[0, p[0]] * auto[0, p[1]]) for p in pairs}
    for c, p in enumerate(pairs):
        assert np.abs(hist[:, c] - gen[:-1, c]).max() < 1e-6 * size[p], p
    np.testing.assert_allclose(k0h, k0g[:-1], rtol=1e-6, atol=1e-7)
    again, _ = pair_products(spectra, pairs, bins, exclude_k0=exclude_k0)
    assert np.array_equal(hist, again)


def test_radial_histogram_special_values():
    """A zero field gives zeros; a field with an infinity gives NaN for its
    pairs alone; a tiny field scales as its square."""
    J, L = 4, 16
    g = torch.Generator(device="cuda").manual_seed(3)
    f = torch.rand((L, L, L), generator=g, device="cuda")
    bad = f.clone()
    bad[1, 2, 3] = float("inf")
    bins = [_win(J, p) for p in KINDS]
    spectra = [rfft_field(x) for x in (torch.zeros_like(f), f, bad, f * 2.0 ** -40)]
    v, _ = pair_products(spectra, [(0, 0), (1, 1), (2, 2), (3, 3)], bins)
    assert np.all(v[:, 0] == 0.0) and np.all(np.isfinite(v[:, 1])) and np.all(np.isnan(v[:, 2]))
    np.testing.assert_array_equal(v[:, 3], v[:, 1] * 2.0 ** -80)


def test_cylindrical_columns_at_bandwidth_two():
    """The folded columns serve every bandwidth: against the generic kernel,
    1e-5 of the largest |value| (the bound of the bandwidth-1 test)."""
    J, L = 5, 32
    g = torch.Generator(device="cuda").manual_seed(5)
    s = [rfft_field(torch.exp(torch.randn((L, L, L), generator=g, device="cuda")))]
    bins = [_win(J, {"type": t, "len_args": {"R": 80.0, "H": 45.0}}, 2) for t in ("ring", "disk", "cylshell", "cylinder")]
    col, _ = pair_products(s, [(0, 0)], bins)
    gen, _ = pair_products(s, [(0, 0)], bins + [_win(J, KINDS[2], 2)])
    assert np.abs(col - gen[:-1]).max() < 1e-5 * np.abs(gen).max()
