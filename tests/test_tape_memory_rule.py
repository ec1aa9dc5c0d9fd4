"""The rule that keeps a whole tape counts the memory that PyTorch's allocator holds without use as free: a
program's cache does not change the route."""

import pytest
import torch

from cmpy_gb300 import adjoint as A


@pytest.mark.parametrize("driver_free,reserved,allocated", [(160, 0, 0), (10, 150, 0), (10, 250, 100), (0, 160, 0)])
def test_cached_memory_is_free(monkeypatch, driver_free, reserved, allocated):
    gb = 1 << 30
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *_: (driver_free * gb, 280 * gb))
    monkeypatch.setattr(torch.cuda, "memory_reserved", lambda *_: reserved * gb)
    monkeypatch.setattr(torch.cuda, "memory_allocated", lambda *_: allocated * gb)
    assert A._tape_spacing(16, gb, 10) == A.TAPE_ALL
    assert A._tape_spacing(16, gb, 11) == 16
