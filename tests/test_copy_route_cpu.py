"""Which copies around a recorded call go through the library's copy kernel (it reads and writes with the current device)."""
import pytest
import torch

from ai2pot_b200 import capi


class _Tensor:
    """What copy_around_call() asks of a tensor: host memory (pinned or not) or memory of a device."""
    def __init__(self, device=None, pinned=False, n=64, dtype=torch.float32, contiguous=True):
        self.device_index, self.pinned, self.n, self.dtype, self.contiguous = device, pinned, n, dtype, contiguous
        self.is_cuda, self.shape, self.copied = device is not None, (n,), False

    numel = lambda self: self.n
    element_size = lambda self: 4
    data_ptr = lambda self: 4096
    is_contiguous = lambda self: self.contiguous
    is_pinned = lambda self: self.pinned
    get_device = lambda self: self.device_index

    def copy_(self, src, non_blocking):
        self.copied = True


@pytest.mark.parametrize("dst,src,kernel", [
    (dict(device=0), dict(pinned=True), True), (dict(pinned=True), dict(device=0), True), (dict(device=0), dict(device=0), True),
    (dict(device=1), dict(pinned=True), False), (dict(pinned=True), dict(device=1), False), (dict(device=0), dict(device=1), False),
    (dict(device=0), dict(), False), (dict(), dict(device=0), False), (dict(device=0, n=1 << 20), dict(pinned=True, n=1 << 20), False),
    (dict(device=0, dtype=torch.float64), dict(pinned=True), False), (dict(device=0), dict(pinned=True, contiguous=False), False)])
def test_route(monkeypatch, dst, src, kernel):
    calls = []

    class Lib:
        def ai2b_chained_copy(self, *a):
            calls.append(a)
            return 0
    monkeypatch.setattr(capi, "lib", Lib)
    monkeypatch.setattr(capi, "_stream", lambda: None)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    d, s = _Tensor(**dst), _Tensor(**src)
    capi.copy_around_call(d, s)
    assert bool(calls) == kernel and d.copied != kernel
