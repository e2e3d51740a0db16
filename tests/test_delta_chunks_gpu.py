"""The gated delta rule in chunks at the sizes where its tiles end: key sizes beside 64 and 128, value columns beside a block's 16
and a warp's 128, portions beside a chunk's 16 tokens, rows without whole 16 bytes; against the plain statement in float64."""

from __future__ import annotations

import pytest
import torch

import pevazen_cases as pc

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("D,Dv", [(12, 1), (16, 15), (63, 17), (65, 136), (127, 129), (128, 256)])
@pytest.mark.parametrize("decay", [-4.0, 2.0])
def test_chunks_at_the_edges_of_tiles(dtype, D, Dv, decay):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    pc.case_delta_rule(dtype, CudaOps(), DEV, H=4, G=2, D=D, Dv=Dv, lens=(15, 16, 17, 31, 33, 64, 3), decay=decay)


def _delta_step(lens, H=4, G=2, D=64, Dv=48, taps=4, seed=0):
    """Random inputs of a step of prompts: the projections x, z and b, and the other arguments of ``delta_rule``."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    T, C = sum(lens), 2 * G * D + H * Dv
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEV)  # noqa: E731
    rand = lambda *shape: torch.randn(shape, generator=g, device=DEV)  # noqa: E731
    x, z, b = rand(T, C).bfloat16(), rand(T, H * D), rand(T, H).bfloat16()
    kw = dict(heads=H, kv_heads=G, dim=D, value_dim=Dv, conv_weight=rand(taps, C), dt_bias=rand(H * D) - 3.0,
              neg_a=-torch.rand(H, generator=g, device=DEV), q_scale=D ** -0.5, cu_seqlens=ints(cu), num_seqs=len(lens),
              positions=ints([i for n in lens for i in range(n)]), token_seq=ints([s for s, n in enumerate(lens) for _ in range(n)]),
              state_slots=ints(list(range(len(lens)))), host_cu_seqlens=cu)
    rings = lambda: torch.zeros((len(lens), taps, C), device=DEV)  # noqa: E731
    states = lambda: torch.ones((len(lens), H, D, Dv), device=DEV) * 0.1  # noqa: E731
    return x, z, b, kw, rings, states


def test_a_step_without_room_for_its_records_runs_token_by_token(monkeypatch):
    from qwen3_runtime_b200.ops.cuda import CudaOps

    ops = CudaOps()
    x, z, b, kw, rings, states = _delta_step([300, 2, 40])
    launched, call, empty = [], ops._call, torch.empty
    records = (342 // 16 + 3) * 4 * 73 * 64

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    def no_room(*size, **options):
        if size == (records,):
            raise torch.OutOfMemoryError("no room")
        return empty(*size, **options)

    monkeypatch.setattr(ops, "_call", spy)
    got = []
    for room in (True, False):
        if not room:
            monkeypatch.setattr(torch, "empty", no_room)
        state = states()
        got.append((ops.delta_rule(x, z, b, ring=rings(), state=state, **kw), state))
    assert [n for n in launched if "scan" in n] == ["q3_delta_chunk_scan", "q3_delta_scan"]
    # float32 sums of a few hundred addends in another order
    for a, c in zip(*got):
        assert float((a - c).abs().max()) <= 3e-5 * float(c.abs().max())


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("what", ["value", "key", "query", "step"])
@pytest.mark.parametrize("D,Dv", [(64, 48), (128, 136), (40, 20)])
def test_what_is_not_finite_leaves_earlier_tokens_alone(what, bad, D, Dv):
    """One input that is no finite number, in the middle of a chunk: the tokens before it, of its chunk too, are as without it, and a
    value's column is the only one that it reaches; as token by token."""
    from qwen3_runtime_b200.ops.cuda import CudaOps

    ops, G, H, at = CudaOps(), 2, 4, 200 + 7
    x, z, b, kw, rings, states = _delta_step([200, 100], H=H, G=G, D=D, Dv=Dv)
    clean = ops.delta_rule(x, z, b, ring=rings(), state=states(), **kw)
    column = {"query": D + 3, "key": G * D + D + 3, "value": 2 * G * D + 3 * Dv + 5}  # of (q | k | v) heads 1, 1 and 3
    if what == "step":
        b[at, 3] = float("nan")
    else:
        x[at, column[what]] = bad
    out = {}
    for chunks in (True, False):
        ops.delta_chunks = chunks
        out[chunks] = ops.delta_rule(x, z, b, ring=rings(), state=states(), **kw)
    heads = [2, 3] if what in ("query", "key") else [3]
    touched = torch.zeros_like(clean, dtype=torch.bool)
    touched[at:, heads, 5 if what == "value" else slice(None)] = True
    for got in out.values():
        # (sums of another order where an infinity stands beside them)
        assert float((got - clean)[~touched].abs().max()) <= 3e-5 * float(clean.abs().max())
        assert not torch.isfinite(got[at][heads][:, 5] if what == "value" else got[at][heads]).any()
