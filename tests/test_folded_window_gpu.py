"""Windows applied from folded tables (and, at J = 9, in the fused x pass)
against the stored per-mode kernel of the same window, and the 512^3 real
transforms against float64.

The folded tables hold the values of the per-mode evaluation; the eight image
terms of a mode are added in another order and the factors multiplied in
another grouping, so each mode differs by at most about 10 roundings of
2^-24 = 6e-7 of it, and the fields by 1e-6 in the 2-norm.  A float32
transform of 512^3 values is off by a few 1e-7 in the 2-norm (log2 N roundings
adding at random): 1e-6."""
import ctypes

import numpy as np
import pytest
import torch

from pyhermes_gb300 import _lib
from pyhermes_gb300.kernels import _ptr, _stream_ptr
from pyhermes_gb300.phi import sample_scaling_function
from pyhermes_gb300.window import WindowFunc, apply_window, rfft_field

pytestmark = pytest.mark.gpu
PHI = sample_scaling_function()
WINDOWS = [({"type": "gaussian", "len_args": {"R": 12.0}}, 1), ({"type": "gaussian", "len_args": {"R": 12.0}}, 2),
           ({"type": "sphere", "len_args": {"R": 20.0}}, 1), ({"type": "shell", "len_args": {"R": 50.0}}, 1),
           ({"type": "thick_shell", "len_args": {"R": 40.0, "delta_R": 10.0}}, 1),
           ({"type": "gaussian_shell", "len_args": {"R_shell": 40.0, "R_smooth": 9.0}}, 1),
           ({"type": "cws", "len_args": {"R": 15.0}}, 1), ({"type": "gdw", "len_args": {"R": 15.0}}, 1),
           ({"type": "laplacian"}, 1), ({"type": "inverse_laplacian"}, 1),
           ({"type": "cylinder", "len_args": {"R": 20.0, "H": 30.0}}, 1),
           ({"type": "ring", "len_args": {"R": 30.0, "H": 8.0}, "kernel_mode": "full_rfft"}, 2),
           ({"type": "disk", "len_args": {"R": 30.0, "H": 8.0}, "los_args": {"nx": 1.0, "ny": 0.0, "nz": 0.0}}, 1),
           ({"type": "sphere", "len_args": {"R": 20.0}}, 2), ({"type": "cubic", "len_args": {"Lx": 9.0, "Ly": 5.0, "Lz": 7.0}}, 1)]


@pytest.mark.parametrize("J", [2, 3, 5, 7, 9])
@pytest.mark.parametrize("k", range(len(WINDOWS)))
def test_folded_window_matches_stored_kernel(J, k):
    p, bw = WINDOWS[k]
    if J == 9 and bw == 2:
        pytest.skip("bandwidth 2 at J = 9 is covered by the smaller levels")
    info = {"J": J, "box_size": 200.0, "phi_resolution": 1024, "wavelet_mode": "db2", "wavelet_level": 10,
            "phi_array": PHI}
    w = WindowFunc(p, info, bandwidth=bw, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(J)
    f = torch.randn((1 << J,) * 3, generator=g, device="cuda")
    got = apply_window(f, w)
    stored = w * 1.0  # a composite: applied from its materialised kernel
    assert stored.materialized and not w.materialized
    ref = apply_window(f, stored)
    assert (got - ref).double().norm() <= 1e-6 * ref.double().norm()


def test_real_transforms_at_512():
    g = torch.Generator(device="cuda").manual_seed(9)
    f = torch.randn((512,) * 3, generator=g, device="cuda")
    ref = torch.fft.rfftn(f.double())
    s = rfft_field(f)
    assert (s - ref).norm() <= 1e-6 * ref.norm()
    del ref
    back = torch.empty_like(f)
    _lib.check(_lib.load().hermes_fft_c2r(_ptr(s), _ptr(back), 9, _stream_ptr(f.device)), "hermes_fft_c2r")
    assert (back / 512 ** 3 - f).double().norm() <= 1e-6 * f.double().norm()


@pytest.mark.parametrize("J,shift", [(6, 0), (9, 0), (9, 8)])
def test_transform_with_a_workspace(J, shift):
    """Own passes (aligned workspace at J = 9) and the plan agree; a workspace
    that is too small is refused."""
    L, lib = 1 << J, _lib.load()
    f = torch.randn((L,) * 3, generator=torch.Generator(device="cuda").manual_seed(J), device="cuda")
    need = ctypes.c_size_t()
    _lib.check(lib.hermes_fft_r2c_workspace_size(J, ctypes.byref(need)), "size")
    ws = torch.empty(need.value + 16, dtype=torch.uint8, device="cuda")[shift:]
    got, ref = (torch.empty((L, L, L // 2 + 1), dtype=torch.complex64, device="cuda") for _ in range(2))
    _lib.check(lib.hermes_fft_r2c_ws(_ptr(f), _ptr(got), J, _ptr(ws), need.value, _stream_ptr(f.device)), "ws")
    _lib.check(lib.hermes_fft_r2c(_ptr(f), _ptr(ref), J, _stream_ptr(f.device)), "plan")
    assert (got - ref).to(torch.complex128).norm() <= 2e-6 * ref.to(torch.complex128).norm()
    if need.value:
        assert lib.hermes_fft_r2c_ws(_ptr(f), _ptr(got), J, _ptr(ws), need.value - 1, _stream_ptr(f.device)) != 0
