"""The float32 product's tile shapes: every one gives the same bits, at sizes that end inside a tile, a slice of K or a
16-byte copy, with rows of wider matrices, and against float64."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 17, 64), (15, 16, 63), (17, 33, 65), (63, 129, 20), (65, 127, 4), (129, 257, 132),
                                   (300, 70, 31)])
@pytest.mark.parametrize("pad", [0, 1, 4])
def test_tile_shapes_give_the_same_bits(ops, M, N, K, pad):
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn((M, K + pad), generator=g).cuda()[:, :K]
    w = torch.randn((N, K + pad), generator=g).cuda()[:, :K]
    want = x.double() @ w.double().t()
    # a chain of K fused additions of products: at most K half units of the running sum of magnitudes
    bound = K * 2.0 ** -24 * float((x.abs().double() @ w.abs().double().t()).max())
    out = []
    try:
        for tile in (-1, 0, 1, 2, 3, 4, 5):
            ops.f32_tile = tile
            out.append(ops.linear(x, w))
    finally:
        ops.f32_tile = -1
    assert float((out[0].double() - want).abs().max()) <= bound
    for other in out[1:]:
        assert torch.equal(out[0], other)


@pytest.mark.parametrize("tile,rows", [(5, 65535 * 16), (3, 65535 * 32), (-1, 65535 * 64)])
def test_more_rows_than_a_grid_has_blocks(ops, tile, rows):
    x = (torch.arange((rows + 3) * 4, device="cuda") % 251).float().view(-1, 4)
    w = torch.tensor([[1.0, 2.0, 3.0, 4.0], [5.0, 0.0, 0.0, 1.0]], device="cuda")
    ops.f32_tile = tile
    try:
        out = ops.linear(x, w)
    finally:
        ops.f32_tile = -1
    for n in range(2):  # sums of small whole numbers are exact
        assert torch.equal(out[:, n], (x * w[n]).sum(1))
