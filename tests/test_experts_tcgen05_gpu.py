"""The routed experts' products on the tcgen05 kernel (csrc/experts_tcgen05.cu) against their torch statement, at the
sizes where its tiles can go wrong: experts with no slot, one, a multiple of 32 and one more or less, a full chunk of 256 and
the first sizes that take two and three; widths that end inside a slice of K or inside a tile of features."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

COUNTS = [0, 1, 31, 32, 33, 0, 255, 256, 257, 512, 513, 2]


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _choices(counts, top, g):
    """``chosen [T, top]`` in which expert e is chosen counts[e] times (padded with a further expert), in random order."""
    slots = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])
    pad = -slots.numel() % top
    slots = torch.cat([slots, torch.full((pad,), len(counts), dtype=torch.int32)])
    return slots[torch.randperm(slots.numel(), generator=g)].view(-1, top).contiguous().cuda()


@pytest.mark.parametrize("width,size", [(64, 64), (72, 136), (320, 88), (128, 392)])
@pytest.mark.parametrize("unit,weight_on,identity", [("clamped_glu", "input", 0), ("clamped_glu", "output", 2), ("relu2", "output", 0)])
def test_products_against_their_statement(ops, width, size, unit, weight_on, identity):
    from emulated_ops import TorchOps

    g = torch.Generator().manual_seed(width + size)
    top = 3
    chosen = _choices(COUNTS, top, g)
    T, stored = chosen.shape[0], len(COUNTS) + 1 - identity
    weights = torch.rand((T, top), generator=g).cuda() + 0.25
    rows = torch.randn((T, width + 16), generator=g).to(torch.bfloat16).cuda()
    h = rows[:, 8: 8 + width]  # rows wider than the layer
    gated = 2 if unit == "clamped_glu" else 1
    first = (width ** -0.5 * torch.randn((stored, gated * size, width), generator=g)).to(torch.bfloat16).cuda()
    down = (size ** -0.5 * torch.randn((stored, width, size), generator=g)).to(torch.bfloat16).cuda()
    shared = torch.randn((T, width), generator=g).to(torch.bfloat16).cuda()
    kw = dict(weight_on=weight_on, shared=shared, activation=unit)
    if unit == "clamped_glu":
        kw.update(limit=1.5, alpha=1.702, up_offset=1.0, num_identity=identity)
    else:
        kw.update(shared_gate=torch.randn((T, 3), generator=g).to(torch.bfloat16).cuda()[:, 1])
    launched = []
    call = ops._call

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    ops._call = spy
    try:
        got = ops.routed_experts(h, chosen, weights, first, down, **kw).float()
    finally:
        del ops._call
    assert launched.count("q3_expert_tcgen05") == 2
    ops.raise_if_kernel_error()
    want = TorchOps().routed_experts(h, chosen, weights, first, down, **kw).float()
    ops.experts_tc = False
    other = ops.routed_experts(h, chosen, weights, first, down, **kw).float()
    ops.experts_tc = True
    # the kernels and the statement round the same places; a product's sum in another order moves a bfloat16 rounding by one unit, 2^-8 of
    # the value, in the expert's hidden row and once more in its output, and the sum over three experts once more
    bound = 3 * 2.0 ** -8 * float(want.abs().max())
    assert float((got - want).abs().max()) <= bound
    assert float((got - other).abs().max()) <= bound


def test_one_token_and_many_experts(ops):
    """Fewer slots than experts, and more tiles than pairs of SMs."""
    from emulated_ops import TorchOps

    g = torch.Generator().manual_seed(5)
    for T, E, width, size in ((1, 40, 64, 64), (700, 200, 256, 264)):
        chosen = torch.stack([torch.randperm(E, generator=g)[:2] for _ in range(T)]).int().cuda()
        weights = torch.rand((T, 2), generator=g).cuda()
        h = torch.randn((T, width), generator=g).to(torch.bfloat16).cuda()
        first = (width ** -0.5 * torch.randn((E, 2 * size, width), generator=g)).to(torch.bfloat16).cuda()
        down = (size ** -0.5 * torch.randn((E, width, size), generator=g)).to(torch.bfloat16).cuda()
        kw = dict(limit=7.0, alpha=1.702, up_offset=1.0, weight_on="input")
        got = ops.routed_experts(h, chosen, weights, first, down, **kw).float()
        ops.raise_if_kernel_error()
        want = TorchOps().routed_experts(h, chosen, weights, first, down, **kw).float()
        assert float((got - want).abs().max()) <= 3 * 2.0 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("tokens,experts,mode", [(1, 5, "sigmoid"), (64, 33, "softmax_chosen"), (65, 64, "sigmoid"), (200, 7, "sigmoid"),
                                                 (130, 256, "softmax_chosen"), (130, 257, "sigmoid")])
def test_router_in_every_batch(ops, tokens, experts, mode):
    """A token's choice and weights are the same bits whatever the batch (few and many tokens take other launch shapes,
    up to 256 outputs another kernel for the choice), and agree with the statement."""
    from emulated_ops import TorchOps

    g = torch.Generator().manual_seed(tokens)
    h = torch.randn((tokens, 136), generator=g).to(torch.bfloat16).cuda()
    router = (0.1 * torch.randn((experts, 136), generator=g)).cuda()
    chosen, weights = ops.route_top(h, router, 5, score=mode)
    want_c, want_w = TorchOps().route_top(h, router, 5, score=mode)
    assert torch.equal(chosen, want_c) and float((weights - want_w).abs().max()) < 1e-5
    for rows in (slice(0, 1), slice(tokens // 2, tokens)):
        c, w = ops.route_top(h[rows], router, 5, score=mode)
        assert torch.equal(c, chosen[rows]) and torch.equal(w, weights[rows])


@pytest.mark.parametrize("counts", [[33, 64, 65, 96, 97, 128], [129, 160, 161, 192, 193, 224], [225, 256, 300, 20, 384, 500]])
@pytest.mark.parametrize("unit", ["clamped_glu", "relu2"])
def test_every_height_of_a_box_of_slots(ops, monkeypatch, counts, unit):
    """Boxes of 32 to 128 rows, an odd and an even number of 32 slots for the two groups of the epilogue."""
    monkeypatch.setitem(globals(), "COUNTS", counts)
    test_products_against_their_statement(ops, 128, 392, unit, "input" if unit == "clamped_glu" else "output", 0)


def _logits(ops, h, router):
    T, E = h.shape[0], router.shape[0]
    logits = torch.empty((T, E), device="cuda")
    chosen, weights = torch.empty((T, 1), dtype=torch.int32, device="cuda"), torch.empty((T, 1), device="cuda")
    ops._call("experts", "q3_route_top", "route_top", 1, h.data_ptr(), h.stride(0), router.data_ptr(), T, E, h.shape[1], 1, 0,
              logits.data_ptr(), chosen.data_ptr(), weights.data_ptr(), None, 0, 0, 0, 1.0)
    return logits


@pytest.mark.parametrize("tokens,experts,width", [(1200, 64, 520), (2400, 33, 136), (400, 200, 72), (40, 20, 100), (33, 20, 37),
                                                  (2500, 17, 2048), (1, 1, 8), (1200, 64, 516), (1200, 64, 36), (300, 33, 4)])
def test_router_logits_of_every_block(ops, tokens, experts, width):
    """Large and small blocks, rows at odd places and widths that end inside a slice: the same bits, near to float64; infinities and
    NaN as float32 products give them, in their own row and column only."""
    g = torch.Generator().manual_seed(tokens + width)
    h = torch.randn((tokens, width), generator=g).to(torch.bfloat16).cuda()
    router = (0.02 * torch.randn((experts, width), generator=g)).cuda()
    got, want = _logits(ops, h, router), h.double() @ router.double().t()
    # a slice's chain of six products rounds six times, then the slices' and the warps' sums, each to 2^-24 of a partial sum
    assert float((got - want).norm() / want.norm()) <= 2.0 ** -24 * (6 + (width / 32) ** 0.5)
    for rows in (slice(0, 1), slice(tokens // 2, tokens)):
        assert torch.equal(_logits(ops, h[rows], router), got[rows])
    odd = torch.zeros((tokens, width + 3), dtype=torch.bfloat16, device="cuda")
    odd[:, 1: 1 + width] = h
    assert torch.equal(_logits(ops, odd[:, 1: 1 + width], router), got)
    if tokens > 3 and experts > 2:
        h[1, width // 2], h[2, 0], router[1, 3] = float("inf"), float("nan"), float("-inf")
        again, want = _logits(ops, h, router), h.double() @ router.double().t()
        assert torch.equal(again.isnan(), want.isnan()) and torch.equal(again.isinf(), want.isinf())
        assert torch.equal(again[again.isinf()], want[want.isinf()].float())
        fine = want.isfinite()
        assert torch.equal(again[fine], got[fine])


@pytest.mark.parametrize("tokens,experts,width", [(1200, 64, 512), (1200, 64, 516), (2400, 33, 40), (40, 20, 100), (1, 5, 8)])
def test_router_logits_of_rows_at_every_place(ops, tokens, experts, width):
    """Loads of 8, 4 and single values, in large and small blocks: the same bits."""
    g = torch.Generator().manual_seed(width)
    h = torch.randn((tokens, width), generator=g).to(torch.bfloat16).cuda()
    router = (0.02 * torch.randn((experts, width), generator=g)).cuda()
    wanted = None
    for pad, first in ((8, 0), (8, 8), (4, 0), (8, 4), (4, 4), (2, 2), (1, 0), (8, 1)):
        rows = torch.full((tokens, width + pad), float("nan"), dtype=torch.bfloat16, device="cuda")
        rows[:, first: first + width] = h
        got = _logits(ops, rows[:, first: first + width], router)
        wanted = got if wanted is None else wanted
        assert torch.equal(got, wanted), (pad, first)
    want = h.double() @ router.double().t()
    assert float((wanted - want).norm() / want.norm()) <= 2.0 ** -24 * (6 + (width / 32) ** 0.5)  # (as above)
