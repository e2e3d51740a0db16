"""Zeroing fixed-size state slots: which slots are zeroed, one fill per cache group whatever the slots, and slots out of range
refused."""

from __future__ import annotations

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from qwen3_runtime_b200.cache.layout import CacheLayout, StateLayerSpec
from qwen3_runtime_b200.cache.storage import CacheStorage

SLOTS = 9


class _Fills(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.count = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        name = func.overloadpacket.__name__
        self.count += name in ("zero_", "fill_", "index_fill_", "copy_") and args[0].dim() > 1
        return func(*args, **(kwargs or {}))


def _storage(device):
    layout = CacheLayout({0: StateLayerSpec((3, 2)), 1: StateLayerSpec((3, 2)), 2: StateLayerSpec((5,))})
    storage = CacheStorage(layout, 16, [], SLOTS, torch.float32, device)
    for t in storage.tensors:
        t.fill_(1.0)
    return storage


DEVICES = [pytest.param("cpu"), pytest.param("cuda", marks=pytest.mark.gpu)]


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("slots", [[4], [3, 4, 5], [8, 0, 5, 2], [7, 1, 1, 7], list(range(0, SLOTS, 2)), [-1, 2]])
def test_one_fill_per_group(device, slots):
    storage = _storage(device)
    with _Fills() as fills:
        storage.zero_state_slots(slots)
    assert fills.count == len(storage.tensors)
    zeroed = {s % (SLOTS + 1) for s in slots}
    for t in storage.tensors:
        for s in range(SLOTS + 1):
            assert bool((t[:, s] == (0.0 if s in zeroed else 1.0)).all()), s


@pytest.mark.parametrize("device", DEVICES)
@pytest.mark.parametrize("slots", [[SLOTS + 1], [0, SLOTS + 1], [3, 400], [-SLOTS - 2]])
def test_slots_out_of_range_are_refused(device, slots):
    storage = _storage(device)
    with pytest.raises(IndexError):
        storage.zero_state_slots(slots)
    assert all(bool((t == 1.0).all()) for t in storage.tensors)
