"""The gated delta rule in chunks at the sizes where its tiles end: key sizes beside 64 and 128, value columns beside a block's 16
and a warp's 128, portions beside a chunk's 16 tokens, rows without whole 16 bytes; against the plain statement in float64."""

from __future__ import annotations

import pytest

import pevazen_cases as pc

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("D,Dv", [(12, 1), (16, 15), (63, 17), (65, 136), (127, 129), (128, 256)])
@pytest.mark.parametrize("decay", [-4.0, 2.0])
def test_chunks_at_the_edges_of_tiles(dtype, D, Dv, decay):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    pc.case_delta_rule(dtype, CudaOps(), DEV, H=4, G=2, D=D, Dv=Dv, lens=(15, 16, 17, 31, 33, 64, 3), decay=decay)
