"""What ``linear_split`` refuses before anything is launched (no device)."""
import pytest
import torch

from bitnet_c_b200.csrc import ops


@pytest.mark.parametrize("w,bias", [("meta", None), ("cpu", "meta")])
def test_operands_on_different_devices_are_refused(monkeypatch, w, bias):
    monkeypatch.setattr(ops, "_need", lambda *a, **k: None)  # (stand-ins for two GPUs)
    x = torch.zeros(32, 256)
    with pytest.raises(ops.KernelError, match="x on cpu, w on"):
        ops.linear_split(x, torch.zeros(128, 256, device=w), None if bias is None else torch.zeros(128, device=bias))
