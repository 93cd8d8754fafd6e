"""Pair products of isotropic bins where the modes that a bin weighs are far
below the largest one: the sums keep what float32 products summed in float64
give.

The reference is the float64 sum of wgt Re(u conj v) K over the same complex64
spectra, with the materialised float32 kernel K.  The windows taken here have
one sign, so no window value cancels: of a product the kernel, T and their
weights are off by a few 2^-24 each (a dozen float32 roundings), 2e-6 of
sum |T K| covers them, and the float64 sums add nothing to that."""
import numpy as np
import pytest
import torch

from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.window import WindowFunc, pair_products, rfft_field

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()


def _windows(J, box=1000.0):
    info = {"J": J, "box_size": box, "phi_resolution": 1024, "wavelet_mode": "db2", "wavelet_level": 10, "phi_array": PHI}
    cell = box / (1 << J)
    return [WindowFunc(p, info, device="cuda") for p in (
        {"type": "gdw", "len_args": {"R": 1.0 * cell}}, {"type": "gdw", "len_args": {"R": 0.6 * cell}},
        {"type": "cw", "len_args": {"R": 0.8 * cell}}, {"type": "laplacian"})]


def _reference(si, sj, win, exclude_k0):
    u, v = si.cpu().numpy().astype(np.complex128), sj.cpu().numpy().astype(np.complex128)
    L = u.shape[0]
    T = (u * np.conj(v)).real * 2.0
    T[:, :, 0] *= 0.5
    T[:, :, L // 2] *= 0.5
    if exclude_k0:
        T[0, 0, 0] = 0.0
    K = np.asarray(win.as_array(), dtype=np.float64)
    return (T * K).sum() / float(L) ** 6, np.abs(T * K).sum() / float(L) ** 6


def _check(spectra, pairs, wins, exclude_k0):
    got, _ = pair_products(spectra, pairs, wins, exclude_k0=exclude_k0)
    for b, w in enumerate(wins):
        for c, (i, j) in enumerate(pairs):
            want, size = _reference(spectra[i], spectra[j], w, exclude_k0)
            assert abs(got[b, c] - want) <= 2e-6 * size, (b, c, got[b, c], want, size)


@pytest.mark.parametrize("J", [3, 5, 6])
def test_weak_contrast_under_a_large_mean(J):
    """A field of mean 1 and contrast 1e-5, its k = 0 mode left in: the largest
    |T| is 10 orders above the modes that W(0) = 0 windows weigh."""
    L = 1 << J
    g = torch.Generator(device="cuda").manual_seed(J)
    s = [rfft_field(1.0 + 1e-5 * torch.randn((L, L, L), generator=g, device="cuda")) for _ in range(2)]
    _check(s, [(0, 0), (0, 1)], _windows(J), False)


@pytest.mark.parametrize("J", [4, 6])
def test_steep_spectrum(J):
    """|u|^2 falling by 16 orders from the box to the Nyquist frequency, under
    windows of the smallest scales."""
    L = 1 << J
    g = torch.Generator(device="cuda").manual_seed(J)
    k = torch.fft.fftfreq(L, device="cuda") * 2.0
    kz = torch.arange(L // 2 + 1, device="cuda") * (2.0 / L)
    kk = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2)
    s = [torch.randn(kk.shape, generator=g, device="cuda", dtype=torch.complex64) * 10.0 ** (-8.0 * kk) * 1e6 for _ in range(2)]
    _check(s, [(0, 0), (1, 1)], _windows(J), True)
