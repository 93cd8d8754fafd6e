"""The fields' z transform inside the prepass and the strided passes (J = 7, 8,
9) against the prepass followed by cuFFT's 3-D plan, for every bin count class,
parity of l and m, degree pairs and a window with a table.  Both transform the
same float32 values; a float32 transform is off by a few 2^-24 sqrt(log2 N) of
the largest value, two of them by at most 2e-6 of max |a|."""
import pytest
import torch

from pyhermes_gb300 import _lib
from pyhermes_gb300 import multipole as mp
from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.window import phi_power_device, rfft_field

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()


@pytest.mark.parametrize("J,nb,l,m", [(7, 1, 0, 0), (7, 4, 3, 1), (7, 5, 4, 2), (7, 16, 5, -3), (8, 2, 2, 1), (8, 8, 7, 7),
                                      (8, 15, 4, 0), (9, 3, 6, 5), (9, 9, 1, 0), (7, 2, 4, "pair"), (8, 9, 0, "pair"),
                                      (9, 6, 8, "pair")])
def test_lines_match_plan(J, nb, l, m):
    L = 1 << J
    g = torch.Generator(device="cuda").manual_seed(10 * J + nb)
    spec = rfft_field(torch.randn((L,) * 3, generator=g, device="cuda"))
    P = phi_power_device(PHI, L, 1, 1024, "cuda")
    radii = [4.0 + 2.5 * i for i in range(nb)]

    def fields():
        if m == "pair":
            return mp.multipole_fields_pair(spec, J, l, radii, P)
        return mp.multipole_fields(spec, J, l, m, radii, P, bin_major=True)

    got = fields()
    assert _lib.load().hermes_multipole_set_fft(0) == 1
    try:
        ref = fields()
    finally:
        _lib.load().hermes_multipole_set_fft(1)
    for b in range(nb):
        x, y = (got[b], ref[b]) if nb > 1 or m == "pair" else (got, ref)
        assert (x - y).abs().max() <= 2e-6 * y.abs().max(), b


def test_lines_with_analytic_bins():
    """The monopole windows' radial table (another table kernel) takes the same route."""
    J, L = 7, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    spec = rfft_field(torch.randn((L,) * 3, generator=g, device="cuda"))
    P = phi_power_device(PHI, L, 1, 1024, "cuda")
    bins = [mp.BinSpec("sphere", {"R": 30.0 + 9 * i}) for i in range(6)]
    got = mp.multipole_fields_bins(spec, J, 0, 0, bins, 1000.0, P, bin_major=True)
    _lib.load().hermes_multipole_set_fft(0)
    try:
        ref = mp.multipole_fields_bins(spec, J, 0, 0, bins, 1000.0, P, bin_major=True)
    finally:
        _lib.load().hermes_multipole_set_fft(1)
    assert (got - ref).abs().max() <= 2e-6 * ref.abs().max()


@pytest.mark.parametrize("J,nb", [(7, 1), (7, 3), (8, 2)])
def test_fields_at_an_odd_complex_value(J, nb):
    """Fields 8 but not 16 bytes aligned: accepted, on the plan's route."""
    L = 1 << J
    g = torch.Generator(device="cuda").manual_seed(J)
    spec = rfft_field(torch.randn((L,) * 3, generator=g, device="cuda"))
    P = phi_power_device(PHI, L, 1, 1024, "cuda")
    radii = [5.0 + 3 * i for i in range(nb)]
    ref = mp.multipole_fields(spec, J, 2, 1, radii, P, bin_major=True).view(-1)
    out = torch.empty(nb * L ** 3 + 2, dtype=torch.complex64, device="cuda")[1:-1]
    assert out.data_ptr() % 16 == 8
    mp.multipole_fields(spec, J, 2, 1, radii, P, out=out, bin_major=True)
    assert (out - ref).abs().max() <= 2e-6 * ref.abs().max()
