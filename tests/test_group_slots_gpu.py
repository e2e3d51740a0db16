"""Grouping slots by expert: one block and two kernels at both sides of the lines between them, with and without the list of
slots, against a count on the host."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("experts", [1, 48, 49, 256, 700])
@pytest.mark.parametrize("slots", [1, 31, 256, 257, 512, 513, 1024, 1025, 5000])
@pytest.mark.parametrize("tile", [32, 256])
def test_every_slot_has_a_place_in_its_experts_group(experts, slots, tile):
    from qwen3_runtime_b200.ops.cuda import CudaOps, _ptr

    ops = CudaOps()
    g = torch.Generator().manual_seed(experts + slots)
    chosen = torch.randint(0, experts, (slots,), generator=g, dtype=torch.int32)
    chosen[: slots // 2] = experts // 2  # one expert with many
    counts = torch.bincount(chosen, minlength=experts)
    first = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    tiles = torch.cat([torch.zeros(1, dtype=torch.long), (-(-counts // tile)).cumsum(0)])
    dev = chosen.cuda()
    need = slots + -(-slots // 1024) * experts
    for scratch_ints in [need] + ([0] if slots <= 512 else []):
        for with_order in (True, False):
            buf = [torch.full((n,), -7, dtype=torch.int32, device="cuda") for n in (experts + 1, experts + 1, slots, slots, need)]
            offsets, tile_offsets, order, place, scratch = buf
            ops._call("experts", "q3_group_slots", "group_slots", _ptr(dev), slots, experts, tile, _ptr(offsets), _ptr(tile_offsets),
                      _ptr(order) if with_order else None, _ptr(place), _ptr(scratch) if scratch_ints else None)
            assert torch.equal(offsets.cpu().long(), first) and torch.equal(tile_offsets.cpu().long(), tiles)
            at = place.cpu().long()
            assert torch.equal(at.sort().values, torch.arange(slots))
            assert bool((at >= first[chosen.long()]).all()) and bool((at < first[chosen.long() + 1]).all())
            if with_order:
                assert torch.equal(order.cpu().long()[at], torch.arange(slots))
            else:
                assert bool((order == -7).all())
