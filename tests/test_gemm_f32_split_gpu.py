"""float32 products on the tensor cores in three bfloat16 parts: nearer to float64 than the FMA chain, a row's bits whatever the
number of rows and the tile, sizes that end inside a tile, a slice or a segment, rows of wider matrices, infinities and NaN."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _matrices(M, N, K, pad=0, positive=False, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + N + K)
    w = torch.randn((N, K + pad), generator=g, device="cuda")[:, :K]
    x = torch.randn((M, K + pad), generator=g, device="cuda")[:, :K]
    return (x.abs(), w.abs()) if positive else (x, w)


@pytest.mark.parametrize("N,K,pad", [(19456, 1032, 0), (2308, 9728, 4), (4100, 4936, 0), (260, 77000, 8), (19500, 1088, 1)])
@pytest.mark.parametrize("positive", [False, True])
def test_nearer_than_the_fma_chain_and_the_same_for_any_rows(ops, N, K, pad, positive):
    x, w = _matrices(337, N, K, pad if pad % 4 == 0 else 0, positive)
    if pad % 4:  # (rows of x without whole 16 bytes; the weights' rows decide who computes)
        x = torch.cat([x, x[:, :pad]], dim=1)[:, :K]
    assert ops._f32_segments(x, w) > 0
    want = x.double() @ w.double().t()
    got = ops.linear(x, w)
    ops.raise_if_kernel_error()
    ops.f32_split = False
    try:
        chain = ops.linear(x, w)
    finally:
        ops.f32_split = True
    error = float((got.double() - want).norm() / want.norm())
    assert error <= float((chain.double() - want).norm() / want.norm())
    # slices of 64 values round towards zero at most 24 times, their sums to nearest: far below a chain's K roundings
    assert error <= 2.0 ** -24 * (6 + (K / 64) ** 0.5)
    for rows in (1, 2, 15, 16, 17, 33, 96, 159, 160, 161, 320, 321):
        assert torch.equal(ops.linear(x[:rows], w), got[:rows]), rows


def test_not_for_weights_it_would_slow_down(ops):
    for N, K in ((2560, 4096), (6144, 2560), (100, 300000), (20000, 1000), (19456, 1028), (19457, 2560)):
        w = torch.empty((N, K), device="cuda")
        assert ops._f32_segments(w[:1], w) == 0, (N, K)
    w = torch.empty((19456, 2561), device="cuda")[:, :2560]
    assert ops._f32_segments(w[:1], w) == 0


def test_infinities_as_float32_gives_them(ops):
    x, w = _matrices(5, 19456, 1088)
    x[1, 7], x[2, 8], x[2, 9] = float("inf"), float("inf"), float("-inf")
    x[3, 1000] = float("nan")
    w[11, 3] = float("-inf")
    w[12, 1087], x[:, 1087] = 3.4e38, 0.5  # (rounds up to infinity in 16 bits; its products do not overflow)
    got, want = ops.linear(x, w), x.double() @ w.double().t()
    ops.raise_if_kernel_error()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got[got.isinf()], want[got.isinf()].float())
    assert torch.equal(got.isinf(), want.float().isinf())


def test_many_rows_in_portions(ops):
    x, w = _matrices(700, 2560, 9728)
    want = ops.linear(x, w)
    ops.F32_SPLIT_ROWS = 256
    try:
        got = torch.full((700, 2570), float("nan"), device="cuda")
        ops.linear(x, w, out=got[:, :2560])
    finally:
        del ops.F32_SPLIT_ROWS
    assert torch.equal(got[:, :2560], want) and bool(got[:, 2560:].isnan().all())


def _times(ops, calls, n=15):
    """Median device time of each call, in turn, behind a cold L2."""
    cold = torch.empty(1 << 26, device="cuda")
    events = [[(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(n)] for _ in calls]
    for call in calls:
        call()
    for i in range(n):
        for call, pairs in zip(calls, events):
            cold.add_(1.0)
            pairs[i][0].record()
            call()
            pairs[i][1].record()
    torch.cuda.synchronize()
    return [sorted(a.elapsed_time(b) for a, b in pairs)[n // 2] for pairs in events]


def test_values_that_are_no_numbers_cost_little_and_stay_with_their_row(ops):
    x, w = _matrices(300, 19456, 2560)
    y, last, v = torch.full_like(x, float("nan")), x.clone(), w.clone()
    last[7, 2559], last[8, 0] = float("nan"), float("inf")
    v[3, 1000] = float("nan")
    finite, one, every, weight = _times(ops, [lambda: ops.linear(x, w), lambda: ops.linear(last, w), lambda: ops.linear(y, w),
                                              lambda: ops.linear(x, v)], 5)
    assert max(one, every, weight) <= 8 * finite, (finite, one, every, weight)
    want = ops.linear(x, w)
    got = ops.linear(last, w)
    keep = [i for i in range(300) if i not in (7, 8)]
    assert got[7].isnan().all() and got[8].isinf().all() and torch.equal(got[keep], want[keep])
    got = ops.linear(x, v)
    assert got[:, 3].isnan().all() and torch.equal(got[:, 4:], want[:, 4:]) and torch.equal(got[:, :3], want[:, :3])
    assert ops.linear(y, w).isnan().all()
    ops.raise_if_kernel_error()


@pytest.mark.parametrize("N,K", [(19456, 2560), (24576, 4096), (8192, 2560), (151936, 2560)])
def test_few_rows_are_no_slower_than_on_the_fma_pipes(ops, N, K):
    x, w = _matrices(32, N, K)

    def fma(rows):
        ops.f32_split = False
        try:
            ops.linear(x[:rows], w)
        finally:
            ops.f32_split = True

    for rows in (1, 16, 32):
        split, chain = _times(ops, [lambda: ops.linear(x[:rows], w), lambda: fma(rows)])
        assert split <= 1.03 * chain, (rows, split, chain)


@pytest.mark.parametrize("N,K", [(19456, 1032), (20480, 1024), (12288, 2048), (2308, 9728)])
def test_few_rows_have_the_bits_of_many(ops, N, K):
    """Items one after another on an SM, whose two halves of warps store unlike numbers of tokens: every number of rows, often."""
    x, w = _matrices(40, N, K)
    want = ops.linear(x, w)
    for rows in range(1, 33):
        for first in (0, 3, 8):
            assert torch.equal(ops.linear(x[first:first + rows], w), want[first:first + rows]), (rows, first)
    ops.raise_if_kernel_error()


def test_scratch_is_bounded_and_gets_smaller_where_there_is_no_room(ops, monkeypatch):
    x, w = _matrices(1000, 24576, 4096)
    want = ops.linear(x[:700], w)
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = ops.linear(x, w)
    assert torch.cuda.max_memory_allocated() - before - got.nbytes <= ops.F32_SPLIT_BYTES + (1 << 20)
    assert torch.equal(got[:700], want)
    empty, asked = torch.empty, []

    def little_room(*size, **options):
        sizes = size[0] if isinstance(size[0], tuple) else size
        if torch.Size(sizes).numel() > 2_000_000 and sizes != (700, 24576):
            asked.append(sizes)
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **options)

    monkeypatch.setattr(torch, "empty", little_room)
    assert torch.equal(ops.linear(x[:700], w), want) and len(asked) > 2
    ops.raise_if_kernel_error()


@pytest.mark.parametrize("sx,sw", [(2.0 ** -100, 1.0), (2.0 ** -118, 1.0), (2.0 ** -126, 1.0), (1.0, 2.0 ** -118), (2.0 ** -64, 2.0 ** -60)])
def test_small_operands_are_off_by_the_smallest_bfloat16_at_most(ops, sx, sw):
    x, w = _matrices(20, 19456, 1088)
    x, w = x * sx, w * sw
    want = x.double() @ w.double().t()
    got = ops.linear(x, w).double()
    ops.raise_if_kernel_error()
    # an operand's parts end at 2^-133: half of that each, times the other operands, beside the error of ordinary operands; results
    # below the normal floats lose up to 2^-149 at every step
    lost = 2.0 ** -134 * (x.double().abs().sum(1)[:, None] + w.double().abs().sum(1)[None, :])
    usual = 2.0 ** -24 * 32 * (x.double().square().sum(1).sqrt()[:, None] * w.double().square().sum(1).sqrt()[None, :])
    assert bool(((got - want).abs() <= lost + usual + 1088 * 2.0 ** -149).all())


def test_products_that_are_left_out_are_below_half_a_digit(ops):
    """Operands just above 1, all alike: their parts' remainders, and so the three products that are left out, have one sign."""
    value = 1.0038987  # parts 1, 2^-8 - ..., with remainders near the largest
    x, w = torch.full((17, 1088), value, device="cuda"), torch.full((19456, 1088), value, device="cuda")
    want = x.double() @ w.double().t()
    error = float(((ops.linear(x, w).double() - want).abs() / want).max())
    # the products left out 2^-24, four large steps of a slice towards zero 2^-23 each, the slices' sums 2^-24 each
    assert error <= 2.0 ** -24 * (1 + 8 + 1088 / 64)


def test_products_that_overflow(ops):
    x, w = torch.zeros((3, 1088), device="cuda"), torch.zeros((19456, 1088), device="cuda")
    w[:, 5], w[:, 70] = 3.0, 3.0
    w[7] = -w[7]
    x[:, 5] = 2e38
    x[1, 70], x[2, 5] = 1e38, 1e38
    got, want = ops.linear(x, w), x.double() @ w.double().t()
    ops.raise_if_kernel_error()
    assert torch.equal(got.isinf(), want.float().isinf()) and not got.isnan().any()
    assert torch.equal(got[got.isinf()], want.float()[got.isinf()])
    finite = ~got.isinf()
    assert torch.allclose(got[finite].double(), want[finite], rtol=1e-6)


@pytest.mark.parametrize("N,K", [(8192, 2560), (20004, 1088), (2564, 8008)])
def test_edges_of_token_tiles_and_of_the_rows_of_a_pair(ops, N, K):
    """Token tiles from one 16 to 160, with four, three and two slices of weights' parts in tensor memory; pairs whose second block
    has few rows or none."""
    x, w = _matrices(481, N, K, 4)
    want = x.double() @ w.double().t()
    whole = ops.linear(x, w)
    for rows in (1, 16, 17, 31, 32, 48, 49, 63, 64, 65, 80, 111, 112, 113, 127, 128, 129, 144, 160, 161, 176, 319, 320, 321, 480):
        got = ops.linear(x[:rows], w)
        ops.raise_if_kernel_error()
        assert torch.equal(got, whole[:rows]), rows
    error = float((whole.double() - want).norm() / want.norm())
    assert error <= 2.0 ** -24 * (6 + (K / 64) ** 0.5)  # (as above)
