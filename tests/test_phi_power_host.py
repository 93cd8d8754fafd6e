"""phi_power_device: the table of every combination is computed once while a
bounded number is in use, however many came before."""
import numpy as np
import torch

from pyhermes_gb300 import window
from pyhermes_gb300.phi import fourier_power_spectrum, sample_scaling_function

PHI = sample_scaling_function()


def test_more_combinations_than_are_kept_on_the_device(monkeypatch):
    calls = []

    def counted(phi, k_max, k_count, res):
        calls.append(k_count)
        return fourier_power_spectrum(phi, k_max, k_count, res)

    monkeypatch.setattr(window, "fourier_power_spectrum", counted)
    monkeypatch.setattr(window, "_POWER_CACHE", {})
    monkeypatch.setattr(window, "_POWER_HOST", type(window._POWER_HOST)())
    n = window._POWER_KEEP + 40
    phis = [PHI * (1.0 + 1e-3 * k) for k in range(n)]
    for p in phis:
        window.phi_power_device(p, 4, 1, 1024, "cpu")
    before = len(calls)
    for p in phis[-8:] * 3:  # what is in use now
        t = window.phi_power_device(p.copy(), 4, 1, 1024, "cpu")
        np.testing.assert_array_equal(t.numpy(), fourier_power_spectrum(p, 1, 4, 1024))
    assert len(calls) == before
    for p in phis * 3:
        window.phi_power_device(p, 4, 1, 1024, "cpu")
    assert len(window._POWER_CACHE) <= window._POWER_KEEP and len(window._POWER_HOST) <= window._POWER_HOST_KEEP


def test_the_table_is_by_value():
    a = window.phi_power_device(PHI, 8, 1, 1024, "cpu")
    assert torch.equal(a, window.phi_power_device(PHI.astype(np.float64).copy(), 8, 1, 1024, torch.device("cpu")))
    assert not torch.equal(a, window.phi_power_device(2.0 * PHI, 8, 1, 1024, "cpu"))
