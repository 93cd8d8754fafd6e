"""The k = 0 coefficient of a field whose coefficients are complex (the result
of a complex window): that of its real part, as the pair products read it."""
import torch

from pyhermes_gb300.corr2pcf import Corr_2PCF
from pyhermes_gb300.sfc_field import SFCField


def test_dc_of_a_complex_field():
    f = SFCField(device="cpu")
    e = torch.rand((4, 4, 4), generator=torch.Generator().manual_seed(1), dtype=torch.float64)
    f.epsilon_device = torch.complex(e, -e).to(torch.complex64)
    assert Corr_2PCF._dc(f) == e.float().double().sum().item()
    f.epsilon_device = e.float()
    assert Corr_2PCF._dc(f) == e.float().double().sum().item()
