"""MultipoleEngine.ddd takes radii as any numbers that float() takes: 0-d and
one-element arrays and tensors beside floats and BinSpecs, equal ones as one bin."""
import numpy as np
import torch

from pyhermes_gb300.multipole import BinSpec, MultipoleEngine


def _engine(bins_seen):
    eng = MultipoleEngine.__new__(MultipoleEngine)
    eng.same23 = True

    def summands_shared(lms, bins):
        bins_seen.append([b.len_args["R"] for b in bins])
        r = np.array(bins_seen[-1])
        return np.array([np.add.outer(r * (1 + l + 10 * m), 100.0 * r) + 0j for l, m in lms])

    eng.summands_shared = summands_shared
    return eng


def test_radii_of_every_kind():
    seen = []
    pairs = [(30.0, 60.0), (np.array(30.0), 60), (torch.tensor(30.0, dtype=torch.float64), np.float64(60.0)),
             (BinSpec("shell", {"R": 30.0}), torch.tensor([60.0])), ("30", np.int64(60))]
    got = _engine(seen).ddd(pairs, 0, 2)
    assert seen == [[30.0, 60.0]]
    want = _engine([]).ddd([(30.0, 60.0)], 0, 2)
    np.testing.assert_array_equal(got, np.repeat(want, len(pairs), axis=0))
