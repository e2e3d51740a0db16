"""The router's choice over logits that are not all finite: NaN comes after every number, lowest index first, and no output
is chosen twice -- the same for up to 256 outputs (logits in registers) and for more (logits in memory)."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _order(row: list[float], top: int) -> list[int]:
    """Numbers in descending order, then NaN; lowest index on a tie."""
    return sorted(range(len(row)), key=lambda e: (math.isnan(row[e]), 0.0 if math.isnan(row[e]) else -row[e], e))[:top]


@pytest.mark.parametrize("outputs", [8, 12, 17, 40, 256, 257, 300])
@pytest.mark.parametrize("tokens", [3, 70, 97])
@pytest.mark.parametrize("mode", [dict(), dict(renormalize=True), dict(score="softmax_chosen")])
def test_choice_with_infinities_and_nan(outputs, tokens, mode):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    ops = CudaOps()
    g = torch.Generator().manual_seed(outputs + tokens)
    # sums of 64 products of small whole numbers over 64: exact in float32, with ties
    h = torch.randint(1, 4, (tokens, 64), generator=g).float()
    router = torch.randint(-8, 9, (outputs, 64), generator=g) / 64.0
    router[[1, outputs // 2, outputs - 1]] = math.nan
    router[[0, 5, outputs - 2]] = -3e38  # sums of 64 such products: minus infinity
    router[7] = 3e38
    h[1] = math.nan  # a token none of whose logits is a number
    logits = h @ router.t()
    for top in (1, 6, outputs - 4, outputs):
        chosen, weights = ops.route_top(h.cuda(), router.cuda(), top, **mode)
        for t in range(tokens):
            assert chosen[t].tolist() == _order(logits[t].tolist(), top), (t, top)
        if not mode:  # the sigmoids; 0 where there is no number
            want = torch.where(logits.isnan(), 0.0, torch.sigmoid(logits)).gather(1, chosen.cpu().long())
            assert float((weights.cpu() - want).abs().max()) <= 1e-6  # a float32 sigmoid


@pytest.mark.parametrize("outputs", [40, 300])
def test_choice_over_all_outputs_stays_in_range(outputs):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    h = torch.ones((5, 64), device="cuda")
    h[2] = math.nan
    router = torch.randn((outputs, 64), generator=torch.Generator().manual_seed(1)).cuda()
    router[3] = math.nan
    chosen, _ = CudaOps().route_top(h, router, 6, score="softmax_all")
    assert 0 <= int(chosen.min()) and int(chosen.max()) < outputs
