"""rfft_field where its workspace cannot be had: the transform without one."""
import pytest
import torch

from pyhermes_gb300 import window

pytestmark = pytest.mark.gpu


def test_without_room_for_the_workspace(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(1)
    f = torch.randn((512, 512, 512), generator=g, device="cuda")
    want = window.rfft_field(f)
    empty, refused = torch.empty, []

    def short(*a, **k):
        if k.get("dtype") == torch.uint8:
            refused.append(a)
            raise torch.OutOfMemoryError("CUDA out of memory.")
        return empty(*a, **k)

    monkeypatch.setattr(torch, "empty", short)
    got = window.rfft_field(f)
    monkeypatch.undo()
    assert refused
    # two float32 transforms of 2^27 values: each is off by 2^-24 sqrt(27) = 3e-7 of the rms (rms), the largest
    # of 7e7 differences by about six times sqrt(2) of that
    rms = want.abs().square().mean().sqrt().item()
    assert (got - want).abs().max().item() < 1e-5 * rms
