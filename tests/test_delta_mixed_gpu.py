"""The gated delta rule over steps that hold prompts and one-token sequences, with the step's lengths given: the prompts in
chunks, the single tokens token by token, against the plain statement in float64."""

from __future__ import annotations

import pytest

import pevazen_cases as pc

pytestmark = pytest.mark.gpu

DEV = "cuda"


class _WithLengths:
    """A kernel table whose delta rule is told the step's lengths, as the part tells it."""

    def __init__(self, ops):
        self.ops, self.launched = ops, []

    def __getattr__(self, name):
        return getattr(self.ops, name)

    def delta_rule(self, *args, **kw):
        call = self.ops._call

        def spy(group, name, what, *a):
            self.launched.append(name)
            return call(group, name, what, *a)

        self.ops._call = spy
        try:
            return self.ops.delta_rule(*args, host_cu_seqlens=kw["cu_seqlens"].tolist(), **kw)
        finally:
            del self.ops._call


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("D,Dv", [(12, 20), (64, 128), (128, 72)])
@pytest.mark.parametrize("lens", [(300,) + (1,) * 4, (1,) * 36 + (160, 1, 17, 16, 2, 31), (1, 70), (40, 33)])
@pytest.mark.parametrize("apart", [True, False])
def test_prompts_beside_single_tokens(dtype, D, Dv, lens, apart):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    ops = _WithLengths(CudaOps())
    ops.ops._delta_long = lambda cu, num_seqs, *_: sum(b - a > 1 for a, b in zip(cu, cu[1:])) if apart else num_seqs
    pc.case_delta_rule(dtype, ops, DEV, D=D, Dv=Dv, lens=lens, decay=-2.5)
    both = apart and 1 in lens
    first = [n for n in ops.launched if n in ("q3_delta_chunk_scan", "q3_delta_scan")][:1 + both]
    assert first == ["q3_delta_chunk_scan"] + ["q3_delta_scan"] * both
