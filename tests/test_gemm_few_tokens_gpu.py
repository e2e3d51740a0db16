"""Products of up to 128 tokens (csrc/gemm_few_tokens.cu) against float64, at the edges of its tiles and of its dispatch."""

import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def draw(M, N, K, seed=1, x_pad=0, w_pad=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K + x_pad, generator=g).to(BF16).cuda()[:, :K]
    w = torch.randn(N, K + w_pad, generator=g).to(BF16).cuda()[:, :K]
    return x, w


def f32_bound(x, w):
    """The products are exact in fp32 and added up in fp32, rounded towards zero at worst: 2^-23 of the sum of magnitudes for each
    of the K / 16 instructions that add to an accumulator, and as much again for the 16 products within one."""
    K = x.shape[1]
    return (x.double().abs() @ w.double().abs().t()) * 2.0**-23 * (K / 16 + 16)


def product(ops, mode, x, w, out, parts=1):
    N = w.shape[0] // (2 if mode >= 2 else 1)
    ops._few_product(mode, x, w, out, parts, x.shape[0], N, x.shape[1])
    ops.raise_if_kernel_error()
    return out


# rows: less than one tile, one row more than a round of 128 rows and of 64, odd; values: one slice, a remainder of 8, odd slices
@pytest.mark.parametrize("N,K", [(1, 8), (3, 64), (296, 72), (18944, 128), (18945, 136), (9473, 320), (2560, 4096)])
@pytest.mark.parametrize("M", [1, 17, 32, 33, 64, 65, 128])
def test_every_mode_against_float64(ops, M, N, K):
    x, w = draw(M, N, K, seed=M + N, x_pad=8, w_pad=16)
    want, bound = x.double() @ w.double().t(), f32_bound(x, w)
    guard = torch.full((M + 1, N + 3), 7.0, device="cuda")
    got = product(ops, 1, x, w, guard[:M, :N])
    assert bool(((got.double() - want).abs() <= bound).all())
    assert bool((guard[M] == 7).all()) and bool((guard[:, N:] == 7).all()), "nothing beyond the result is written"
    rounded = product(ops, 0, x, w, torch.empty((M, N), dtype=BF16, device="cuda"))
    assert torch.equal(rounded, got.to(BF16))
    parts = ops._get("gemm_few_tokens", "q3_gemm_few_parts")(M, N, K, 8)
    if parts > 1:
        planes = product(ops, 1, x, w, torch.full((parts, M, N), 7.0, device="cuda"), parts)
        assert bool(((planes.double().sum(0) - want).abs() <= bound).all())
    if N > 1:
        I = N // 2
        for mode, act in ((2, "silu"), (3, "gelu")):
            unit = product(ops, mode, x, w[: 2 * I], torch.empty((M, I), dtype=BF16, device="cuda"))
            sums = product(ops, 1, x, w[: 2 * I].contiguous(), torch.empty((M, 2 * I), device="cuda"))
            want_unit = ops.glu_mul(sums, torch.empty((M, I), device="cuda"), act).to(BF16)
            assert torch.equal(unit, want_unit), "the unit takes the fp32 products"


@pytest.mark.parametrize("N,K,parts", [(24576, 256, 1), (1024, 328, 1), (24576, 896, 1), (24576, 2560, 1), (10240, 5120, 1),
                                       (4096, 12288, 8)])
@pytest.mark.parametrize("M", [1, 9, 16])
@pytest.mark.parametrize("positive", [False, True])
def test_sums_of_up_to_16_tokens_are_as_near_as_the_streams(ops, monkeypatch, M, N, K, parts, positive):
    """The streaming kernels add 16 chains of a sixteenth of K each; one chain over all of K would be an order of magnitude further
    off, most of all where nothing cancels."""
    x, w = draw(M, N, K, seed=K + M)
    if positive:
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().t()
    if parts > 1:
        parts = ops._get("gemm_few_tokens", "q3_gemm_few_parts")(M, N, K, parts)
        assert parts > 1
    got = product(ops, 1, x, w, torch.empty((parts, M, N), device="cuda"), parts).sum(0)
    monkeypatch.setattr(ops, "small_gemm", "stream")
    other = ops.linear(x, w, partial_sums=True) if parts > 1 else ops.linear(x, w, out_dtype=F32)
    off = lambda y: float((y.double() - want).norm() / want.norm())
    assert off(got) <= off(other.sum(0) if parts > 1 else other)
    # two instructions to an accumulator, rounded towards zero, and 16 products within one (as f32_bound); then roundings to nearest:
    # three on the way of eight accumulators, one of each eight, one of each plane
    bound = (x.double().abs() @ w.double().abs().t()) * 2.0**-24 * (2 * (2 + 16) + 3 + K / 256 + parts)
    assert bool(((got.double() - want).abs() <= bound).all())


# what linear and gated_linear send here and what they do not
@pytest.mark.parametrize("M", [16, 17, 32, 33, 64, 65, 128, 129])
@pytest.mark.parametrize("pad", [0, 8, 4])
def test_routes_agree(ops, M, pad):
    x, w = draw(M, 24577, 512, seed=M, x_pad=pad, w_pad=pad)
    want = x.double() @ w.double().t()
    before = ops.launches
    got = ops.linear(x, w, out_dtype=F32)
    assert bool(((got.double() - want).abs() <= f32_bound(x, w)).all())
    assert (ops.launches > before) == (M <= 128 and pad % 8 == 0)
    out = torch.empty((M, 24577), device="cuda")
    assert ops.linear(x, w, out=out, out_dtype=F32) is out and torch.equal(out, got)
    x, w = draw(M, 1024, 3072, seed=M + 1, x_pad=pad, w_pad=pad)
    want = x.double() @ w.double().t()
    planes = ops.linear(x, w, partial_sums=True)
    if planes.dim() == 3:  # (the library's product of rows off 16 bytes may add its own ranges up in bfloat16)
        assert bool(((planes.double().sum(0) - want).abs() <= f32_bound(x, w)).all())
    if 16 < M <= 128:
        assert (planes.dim() == 3) == (M <= 64 and pad % 8 == 0)
    x, w = draw(M, 2 * 5008, 2048, seed=M + 2, x_pad=pad, w_pad=pad)
    w = w * 0.02
    got = ops.gated_linear(x, w, torch.empty((M, 5008), dtype=BF16, device="cuda"))
    sums = (x.double() @ w.double().t()).to(BF16).double()
    gate, up = sums[:, :5008], sums[:, 5008:]
    want = gate * torch.sigmoid(gate) * up
    # gate and up are off by their fp32 sums and may be rounded to the neighbouring bfloat16 (2^-8 of them), the unit's slope in
    # the gate is at most 1.1, and the result is rounded once more
    off = f32_bound(x, w)
    off_gate, off_up = off[:, :5008] + 2.0**-8 * gate.abs(), off[:, 5008:] + 2.0**-8 * up.abs()
    bound = 1.1 * (off_gate * (up.abs() + off_up) + off_up * gate.abs()) + 2.0**-8 * want.abs() + 1e-12
    if pad % 8 == 0 or M <= 16:
        assert bool(((got.double() - want).abs() <= bound).all())


def large(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(BF16)
    return x, (0.02 * torch.randn((N, K), generator=g, device="cuda")).to(BF16)


def launched(ops, monkeypatch, call):
    """The result of ``call()`` and the modes in which it launched this file's kernel."""
    modes, under = [], ops._call

    def spy(group, name, what, *args):
        modes.extend(args[:1] if name == "q3_gemm_few_tokens" else [])
        return under(group, name, what, *args)

    monkeypatch.setattr(ops, "_call", spy)
    result = call()
    monkeypatch.undo()
    ops.raise_if_kernel_error()
    return result, modes


# both sides of every line of CudaOps.FEW_TOKENS: tokens, rows, values, result, whether it is this kernel's
@pytest.mark.parametrize("M,N,K,dtype,taken", [
    (1, 24576, 64, F32, True), (16, 24568, 64, F32, False), (16, 24576, 64, BF16, True), (17, 24576, 64, BF16, True),
    (17, 24568, 64, F32, False), (64, 24576, 64, BF16, True), (65, 24576, 64, BF16, False), (128, 24576, 64, F32, True),
    (129, 24576, 64, F32, False), (16, 10240, 5080, BF16, True), (16, 10240, 5072, BF16, False), (16, 10232, 5088, BF16, False),
    (1, 10240, 5080, F32, True), (17, 10240, 5080, F32, False), (16, 20480, 2560, BF16, False), (16, 20480, 2568, BF16, True),
    (9, 16384, 4088, BF16, True), (8, 16384, 4088, BF16, False), (8, 16384, 4096, BF16, True), (8, 18944, 2752, BF16, False),
    (8, 18952, 2752, BF16, True)])
def test_which_finished_products_are_taken(ops, monkeypatch, M, N, K, dtype, taken):
    x, w = large(M, N, K)
    got, modes = launched(ops, monkeypatch, lambda: ops.linear(x, w, out_dtype=dtype))
    assert modes == [int(dtype == F32)] * taken and got.dtype == dtype
    want = x.double() @ w.double().t()
    assert bool(((got.double() - want).abs() <= f32_bound(x, w) + (2.0**-8 * want.abs() if dtype == BF16 else 0)).all())


@pytest.mark.parametrize("M,N,K,taken", [
    (16, 3664, 12288, True), (16, 3656, 12288, False), (16, 3680, 12280, False), (1, 3664, 12288, True), (16, 4096, 13056, True),
    (16, 4096, 13064, False), (16, 4096, 16888, False), (16, 4096, 16896, True), (16, 4088, 16896, False), (9, 2200, 20480, False),
    (9, 2200, 20488, True), (9, 2192, 20488, False), (17, 1024, 3072, True),
    (17, 1024, 3064, False), (17, 4096, 12288, True), (17, 4104, 12288, False), (64, 1024, 3072, True), (65, 1024, 3072, False)])
def test_which_partial_sums_are_taken(ops, monkeypatch, M, N, K, taken):
    x, w = large(M, N, K)
    got, modes = launched(ops, monkeypatch, lambda: ops.linear(x, w, partial_sums=True))
    assert modes == [1] * taken
    want, bound = x.double() @ w.double().t(), f32_bound(x, w)
    if got.dim() == 3:
        got = got.double().sum(0)
    else:
        assert not taken
        bound = bound + 2.0**-8 * want.abs()
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M,I,K,taken", [
    (1, 9768, 4096, True), (16, 9768, 4096, True), (16, 9760, 4096, False), (17, 2448, 4096, True), (17, 2440, 4096, False),
    (32, 2448, 4096, True), (33, 2448, 4096, False), (33, 16384, 64, True), (33, 16376, 64, False), (64, 16384, 64, True),
    (65, 16384, 64, False)])
@pytest.mark.parametrize("act", ["silu", "gelu"])
@pytest.mark.parametrize("aligned", [True, False])
def test_which_gated_products_are_taken(ops, monkeypatch, M, I, K, taken, act, aligned):
    x, w = large(M, 2 * I, K)
    if not aligned:  # rows at odd multiples of 8 bytes: never this kernel's
        x = torch.nn.functional.pad(x, (0, 4))[:, :K]
    got, modes = launched(ops, monkeypatch, lambda: ops.gated_linear(x, w, torch.empty((M, I), dtype=BF16, device="cuda"), act))
    assert (modes == [2 + (act == "gelu")]) == (taken and aligned) and (aligned or not modes)
    sums = x.double() @ w.double().t()
    gate, up = sums[:, :I], sums[:, I:]
    unit = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    want = unit * up
    # gate and up are off by their fp32 sums and may be rounded to the neighbouring bfloat16 (2^-8 of them); where the library takes
    # rows off 16 bytes, it may cut K and round the ranges' sums and their additions, each at most the sum of magnitudes, as well (16
    # ranges: 16 x 2^-8).  The unit's slope in the gate is at most 1.13, and the result is rounded once more.
    magnitudes = x.double().abs() @ w.double().abs().t()
    off = f32_bound(x, w) + 2.0**-8 * sums.abs() + (0 if aligned else 16 * 2.0**-8 * magnitudes)
    bound = 1.13 * (off[:, :I] * (up.abs() + off[:, I:]) + off[:, I:] * gate.abs()) + 2.0**-8 * want.abs() + 1e-12
    assert bool(((got.double() - want).abs() <= bound).all())


def test_sizes_settle_most_calls(ops, monkeypatch):
    """Strides, types and alignment are looked at only where the sizes are this kernel's: a call that is not pays for comparisons."""
    monkeypatch.setattr(ops, "_few_tokens_ok", lambda x, weight: pytest.fail("asked for"))
    for M in (1, 16, 17, 64, 128, 129, 300):
        x, w = draw(M, 256, 264)
        for kw in ({}, dict(partial_sums=True), dict(out_dtype=F32)):
            ops.linear(x, w, **kw)
        ops.gated_linear(x, w, torch.empty((M, 128), dtype=BF16, device="cuda"))


def test_weights_the_kernel_before_writes_and_a_captured_step(ops):
    M, N, K = 48, 24576, 256
    x, w = draw(M, N, K)
    sources = [draw(M, N, K, seed=2 + i)[1] for i in range(4)]
    weight, got = torch.zeros_like(w), []
    for src in sources:
        weight.copy_(src)
        got.append(ops.linear(x, weight, out_dtype=F32))
    for src, y in zip(sources, got):
        assert torch.equal(y, ops.linear(x, src, out_dtype=F32)), "same sums in the same order"
    out = torch.empty((M, N), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.linear(x, weight, out=out, out_dtype=F32)
    for src, y in zip(sources, got):
        weight.copy_(src)
        graph.replay()
        assert torch.equal(out, y)
    ops.raise_if_kernel_error()
