"""The contraction of few bins, several tiles side by side in one block,
against the 16-bin form of the same kernel (the same fields padded to more
than 8 bins).  Every tile keeps its operands and their order, and the tiles
are added in the same order: the same bits."""
import ctypes

import numpy as np
import pytest
import torch

from pyhermes_gb300 import multipole as mp
from pyhermes_gb300.phi import cal_gamma, sample_scaling_function

pytestmark = pytest.mark.gpu
GAMMA = (ctypes.c_double * 9)(*cal_gamma(sample_scaling_function(), 3, 1024).ravel())


def _contract(eps, f2, nb2, J, f3=None, nb3=None, conj_sign=1, packed=False):
    out = torch.zeros((16, 16, 2), dtype=torch.float64, device="cuda")
    if packed:
        mp.multipole_contract_pair_async(eps, f2, nb2, GAMMA, J, out)
    else:
        mp.multipole_contract_async(eps, f2, nb2, GAMMA, J, out, fields3=f3, nb3=nb3, conj_sign=conj_sign, bin_major=True)
    assert mp.contract_status(J) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("J", [4, 5, 6, 7])
@pytest.mark.parametrize("nb2,nb3", [(1, 0), (2, 0), (3, 0), (4, 0), (5, 0), (8, 0), (2, 1), (3, 7), (4, 2)])
def test_tiles_match_single_tile(J, nb2, nb3):
    N = 1 << (3 * J)
    g = torch.Generator(device="cuda").manual_seed(100 * J + 10 * nb2 + nb3)
    eps = torch.randn((1 << J,) * 3, generator=g, device="cuda")

    def fields(nb):
        return torch.view_as_complex(torch.randn((nb, N, 2), generator=g, device="cuda"))

    def padded(f):
        return torch.cat([f, torch.zeros((9 - f.shape[0], N), dtype=f.dtype, device="cuda")])

    f2 = fields(nb2)
    if nb3:
        f3 = fields(nb3)
        got, ref = _contract(eps, f2, nb2, J, f3, nb3), _contract(eps, padded(f2), 9, J, padded(f3), 9)
        assert np.array_equal(got[:nb2, :nb3], ref[:nb2, :nb3])
        return
    for kw in ({"conj_sign": 1}, {"conj_sign": -1}, {"packed": True}):
        got, ref = _contract(eps, f2, nb2, J, **kw), _contract(eps, padded(f2), 9, J, **kw)
        assert np.array_equal(got[:nb2, :nb2], ref[:nb2, :nb2]), kw
        assert np.all(got[nb2:] == 0) and np.all(got[:, nb2:] == 0)
