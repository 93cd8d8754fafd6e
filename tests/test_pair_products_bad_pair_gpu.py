"""A spectrum that is not finite spoils its own pairs and no other: the finite
pairs of the same call have the values that they have beside a finite field in
its place, bit for bit, whatever their number and the bad pair's place.  (The
radial bins' histograms are exact sums of their own pair, so they also equal a
call of that pair alone; the cylindrical pass takes the columns of one pair in
other groups than those of several.)"""
import numpy as np
import pytest
import torch

from pyhermes_gb300.corr2pcf import Corr_2PCF
from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.sfc_field import SFCField
from pyhermes_gb300.window import WindowFunc, pair_products, rfft_field

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()
J, L = 5, 32
INFO = {"J": J, "box_size": 1000.0, "phi_resolution": 1024, "wavelet_mode": "db2", "wavelet_level": 10, "phi_array": PHI}
BINS = {"radial": ({"type": "shell", "len_args": {"R": 0.0}}, {"type": "sphere", "len_args": {"R": 70.0}},
                   {"type": "gaussian", "len_args": {"R": 25.0}}),
        "cylindrical": ({"type": "ring", "len_args": {"R": 80.0, "H": 45.0}},
                        {"type": "ring", "len_args": {"R": 20.0, "H": 10.0}}),
        "generic": ({"type": "shell", "len_args": {"R": 40.0}},
                    {"type": "cubic", "len_args": {"Lx": 30.0, "Ly": 20.0, "Lz": 10.0}})}


def _values(k):
    g = torch.Generator(device="cuda").manual_seed(k)
    return torch.exp(torch.randn((L, L, L), generator=g, device="cuda"))


def _spoilt(x, value):
    x = x.clone()
    x[1, 2, 3] = value
    return x


@pytest.mark.parametrize("kind", sorted(BINS))
@pytest.mark.parametrize("n_pairs", [2, 3, 4])
def test_finite_pairs_beside_a_bad_one(kind, n_pairs):
    bins = [WindowFunc(p, INFO, device="cuda") for p in BINS[kind]]
    good = [rfft_field(_values(k)) for k in range(4)]
    for at in range(n_pairs):
        pairs = [(0, 0), (0, 1), (2, 1), (2, 2)][:n_pairs]
        pairs[at] = (3, 3) if at % 2 else (1, 3)
        want, _ = pair_products(good, pairs, bins)
        for value in (float("inf"), float("nan")):
            v, _ = pair_products(good[:3] + [rfft_field(_spoilt(_values(3), value))], pairs, bins)
            assert np.all(np.isnan(v[:, at]))
            for c in set(range(n_pairs)) - {at}:
                assert np.all(v[:, c] != 0.0) and np.array_equal(v[:, c], want[:, c]), (at, c)
                if kind == "radial":
                    assert np.array_equal(v[:, c], pair_products(good, [pairs[c]], bins)[0][:, 0]), (at, c)


def test_tiny_fields_scale_as_their_square():
    bins = [WindowFunc(p, INFO, device="cuda") for p in BINS["radial"]]
    f = _values(1)
    v, _ = pair_products([rfft_field(f), rfft_field(f * 2.0 ** -40)], [(0, 0), (1, 1)], bins)
    assert np.all(v != 0.0)
    np.testing.assert_array_equal(v[:, 1], v[:, 0] * 2.0 ** -80)


def test_data_products_beside_a_bad_random_field():
    """Corr_2PCF: dd of a finite data field, with a random field that holds an
    infinity, is the dd of a run without it."""
    def field(eps):
        f = SFCField(threads=1, device="cuda")
        f.sfc_info = {"particle_count": 1000, "catalog_weight_sum": 1.0, "catalog_weight_sq_sum": 1.0,
                      "raw_field_weighted_sum": 1.0, "field_integral": float(eps.double().sum().item()),
                      "L": L, "V": L ** 3, "scale_factor": L / 1000.0, "field_kind": "catalog_field",
                      "weight_normalization": "catalog", "phi_support": 3, "fin": {}, "particle_data_retrievable": False,
                      "particle_data_path": "", "particle_data_format": "", **INFO}
        f.format_sfc_params()
        f.epsilon_device = eps
        return f

    p = {"sfc_field": field(_values(1)), "sampling": {"s": [0.0, 40.0, 90.0]}}
    want = Corr_2PCF({"Corr_2PCF": {**p, "products": ["dd"]}}).run(save_result=False).dd
    r = field(_spoilt(_values(2), float("inf")))
    got = Corr_2PCF({"Corr_2PCF": {**p, "random": r, "products": ["dd", "rr"]}}).run(save_result=False)
    np.testing.assert_array_equal(got.dd, want)
    assert not np.any(np.isfinite(got.rr))
