"""Which stream the bindings ask for, on the CPU with stand-ins for torch's calls: the current device's for launches, the tensor's own
device's for scratch, and both without torch's internal short cut."""
from types import SimpleNamespace

import pytest
import torch

from zipage_b200 import _lib as L
from zipage_b200.layers import attention as A


@pytest.fixture(params=["number", "object"])
def streams(request, monkeypatch):
    """Device 2 is the current one; device i's current stream is 100 + i."""
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 2)
    objects = []
    if request.param == "number":
        monkeypatch.setattr(L, "_raw_stream", lambda i: 100 + i)
    else:
        monkeypatch.setattr(L, "_raw_stream", None)

    def current_stream(device=None):
        objects.append(device)
        return SimpleNamespace(cuda_stream=100 + (2 if device is None else device))
    monkeypatch.setattr(torch.cuda, "current_stream", current_stream)
    yield objects
    assert request.param == "object" or not objects      # (no Stream object where the number is to be had)


def test_launches_go_to_the_current_devices_stream(streams):
    assert L.stream_ptr() == 102


def test_scratch_belongs_to_the_stream_of_the_tensors_device(streams, monkeypatch):
    monkeypatch.setattr(A, "_ws_cache", {})
    monkeypatch.setattr(A, "_ws_kept", [])
    monkeypatch.setattr(torch, "empty", lambda n, dtype, device: SimpleNamespace(numel=lambda: n, device=device))
    device = torch.device("cuda", 1)
    buf = A._workspace(device, 100)
    assert list(A._ws_cache) == [(1, 101)] and buf.device == device
    assert A._workspace(device, 1 << 20) is buf
    bigger = A._workspace(device, (1 << 20) + 1)
    assert A._ws_kept == [buf] and A._ws_cache == {(1, 101): bigger}
    assert A._workspace(torch.device("cuda", 2), 1) is not bigger
