"""The fields that a task prepares are its own: an edit in place of one vertex,
of the reference field or of the input acts on that one alone, whether the
vertices came from one input or from several."""
import copy

import numpy as np
import pytest
import torch

from pyhermes_gb300.corr2pcf import Corr_2PCF
from pyhermes_gb300.multipole import Corr_3PCF_Multipole
from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.sfc_field import SFCField

L = 8


def _field(seed, kind="catalog_field", norm="catalog"):
    eps = torch.rand((L, L, L), generator=torch.Generator().manual_seed(seed))
    f = SFCField(threads=1, device="cpu")
    f.sfc_info = {"particle_count": 1000, "catalog_weight_sum": 2.0, "catalog_weight_sq_sum": 1.0,
                  "raw_field_weighted_sum": 4.0, "field_integral": float(eps.double().sum().item()),
                  "J": 3, "box_size": 1000.0, "L": L, "V": L ** 3, "scale_factor": L / 1000.0, "field_kind": kind,
                  "weight_normalization": norm, "phi_support": 3, "phi_resolution": 1024, "wavelet_mode": "db2",
                  "wavelet_level": 10, "phi_array": sample_scaling_function(), "fin": {},
                  "particle_data_retrievable": False, "particle_data_path": "", "particle_data_format": ""}
    f.format_sfc_params()
    f.epsilon_device = eps
    return f


def _two(products):
    return Corr_2PCF({"Corr_2PCF": {"sfc_field": _field(1), "random": _field(2), "sampling": {"s": [100.0]},
                                    "products": products}}, device="cpu"), (1, 2)


def _three(products):
    w = {"type": "shell", "len_args": {}, "other_args": {}}
    return Corr_3PCF_Multipole({"Corr_3PCF_Multipole": {
        "sfc_field": _field(1), "random": _field(2), "binning_window12": {**w, "mapping": {"R": "r12"}},
        "binning_window13": {**w, "mapping": {"R": "r13"}}, "sampling": {"mode": "paired", "r12": [150.0], "r13": [250.0]},
        "l_min": 0, "l_max": 1, "summation_backend": "gb300", "products": products}}, device="cpu"), (1, 2, 3)


def _set(task, n, data, rand):
    for i in range(1, n + 1):
        setattr(task, f"sfc_field{i}", data[min(i, len(data)) - 1])
        setattr(task, f"random{i}", rand[min(i, len(rand)) - 1])


@pytest.mark.parametrize("make,products", [(_two, ["dd", "rr"]), (_three, ["delta_ddd_l"])])
@pytest.mark.parametrize("kind,norm", [("catalog_field", "catalog"), ("catalog_field", "raw"), ("derived_field", None)])
@pytest.mark.parametrize("inputs", ["one", "each"])
def test_an_edit_acts_on_one_field(make, products, kind, norm, inputs):
    task, vertices = make(products)
    n = len(vertices)
    m = 1 if inputs == "one" else n
    data = [_field(10 + i, kind, norm) for i in range(m)]
    rand = [_field(20 + i, kind, norm) for i in range(m)]
    _set(task, n, data, rand)
    task.prepare_input_fields()
    owned = [task.data[i] for i in vertices] + [task.rand[i] for i in vertices]
    owned += [task.reference] if hasattr(task, "reference") else []
    fields = owned + data + rand
    values = [f.epsilon_device.clone() for f in fields]
    # and a second look gives the same tensor
    assert all(f.epsilon_device is f.epsilon_device for f in fields)
    for k, f in enumerate(fields):
        f.epsilon_device.add_(k + 1.0)
        values[k] += k + 1.0
        for v, h in zip(values, fields):
            assert torch.equal(h.epsilon_device, v)


def test_edits_of_arrays_and_copies():
    """The host array, deep copies and derived fields share nothing either."""
    f = _field(5) * 2.0  # nobody holds its tensor
    a, b = f._snapshot(), f._snapshot()
    assert a._coefficients() is b._coefficients() is f._coefficients()
    c = copy.deepcopy(a)
    want = f.epsilon.copy()
    for k, h in enumerate((a, b, c, f)):
        h.epsilon[0, 0, 0] = 100.0 + k
        h.epsilon_device[1, 1, 1] = 50.0 + k
    for k, h in enumerate((a, b, c, f)):
        got = h.epsilon_device.double().numpy().copy()
        assert got[1, 1, 1] == 50.0 + k and got[0, 0, 0] in (100.0 + k, want[0, 0, 0])
        got[1, 1, 1], got[0, 0, 0] = want[1, 1, 1], want[0, 0, 0]
        np.testing.assert_array_equal(got, want)
    held = _field(6)
    assert held._snapshot()._coefficients() is not held._coefficients()


def test_a_float64_array_keeps_its_digits():
    f = _field(7)
    f.epsilon = f.epsilon + 1e-12
    task, _ = _two(["dd"])
    task.sfc_field1 = task.sfc_field2 = f
    task.prepare_input_fields()
    for i in (1, 2):
        np.testing.assert_array_equal(task.data[i].epsilon, f.epsilon)
        assert task.data[i].epsilon is not f.epsilon


@pytest.mark.parametrize("make,products", [(_two, ["dd", "rr"]), (_three, ["delta_ddd_l"])])
def test_an_edit_of_the_input_after_the_preparation(make, products):
    """A tensor of the input that the caller took before the preparation."""
    task, vertices = make(products)
    data, rand = _field(3), _field(4)
    held = [data.epsilon_device, rand.epsilon_device]
    _set(task, len(vertices), [data], [rand])
    task.prepare_input_fields()
    kept = [task.data[i].epsilon.copy() for i in vertices] + [task.rand[i].epsilon.copy() for i in vertices]
    for t in held:
        t.mul_(7.0)
    assert data.epsilon_device is held[0] and rand.epsilon_device is held[1]
    now = [task.data[i].epsilon_device for i in vertices] + [task.rand[i].epsilon_device for i in vertices]
    for a, b in zip(kept, now):
        np.testing.assert_array_equal(a, b.double().numpy())
