"""The row ops launch on the device of their tensors and on a stream of it, whichever device is current, and refuse
arguments on another one.  (Recorders stand in for the device context, the stream and the library.)"""
import pytest
import torch

from wsvd_b200 import ops


@pytest.fixture
def log(monkeypatch):
    seen = []

    class Guard:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            seen.append(f"enter {self.device}")

        def __exit__(self, *_):
            seen.append("exit")

    class Library:
        def __getattr__(self, name):
            return lambda *args: seen.append(name) or 0

    monkeypatch.setattr(ops, "_on_device", Guard)
    monkeypatch.setattr(ops, "_stream", lambda stream: seen.append("stream"))
    monkeypatch.setattr(ops, "_cuda_tensor", lambda *args, **kw: None)
    monkeypatch.setattr(ops._lib, "lib", lambda: Library())
    return seen


def _calls(other):
    """Each op with its further arguments on the device `other`."""
    x = torch.zeros(4, 8, dtype=torch.float16)
    y = torch.zeros(4, 8, dtype=torch.float16, device=other)
    q = torch.zeros(2, 3, 8, dtype=torch.float16)
    pos, freq = torch.zeros(2, dtype=torch.int32, device=other), torch.zeros(4, device=other)
    return {
        "wsvd_rms_norm_f16": lambda: ops.rms_norm(x, out=y),
        "wsvd_add_rms_norm_f16": lambda: ops.add_rms_norm(x, y),
        "wsvd_rope_half_f16": lambda: ops.rope_half_(q, pos, freq),
        "wsvd_silu_mul_f16": lambda: ops.silu_mul(x, y),
    }


@pytest.mark.parametrize("name", list(_calls("cpu")))
def test_the_tensors_device_is_entered(log, name):
    _calls("cpu")[name]()
    assert log in (["enter cpu", "stream", name, "exit"], ["enter cpu", name, "stream", "exit"])


@pytest.mark.parametrize("name", list(_calls("cpu")))
def test_two_devices_are_refused(log, name):
    with pytest.raises(ValueError, match="is on meta, expected cpu"):
        _calls("meta")[name]()
    assert not log


def test_the_device_context_is_entered_only_where_it_is_not_in_place(monkeypatch):
    entered = []
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(torch.cuda, "device", lambda d: entered.append(d.index))
    ops._on_device(torch.device("cuda", 0))
    assert entered == []
    ops._on_device(torch.device("cuda", 1))
    assert entered == [1]
