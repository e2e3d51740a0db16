"""The chunks of the decayed state scan (csrc/linear_state.cu) where they can go wrong: portions of a chunk more or less one
token, segments of one chunk and of several, value columns that fill no tile, values that are not finite."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _step(lens, H, D, Dv, seed=0):
    g = torch.Generator().manual_seed(seed)
    T, cu = sum(lens), [0]
    for n in lens:
        cu.append(cu[-1] + n)
    q, k, z = (torch.randn((T, H, D), generator=g).bfloat16().cuda() for _ in range(3))
    v = torch.randn((T, H, Dv), generator=g).bfloat16().cuda()
    kw = dict(cu_seqlens=torch.tensor(cu, dtype=torch.int32, device="cuda"), num_seqs=len(lens), decay_logits=z, tau=4.0,
              state_slots=torch.arange(len(lens), dtype=torch.int32, device="cuda"), host_cu_seqlens=cu, q_scale=0.25)
    return q, k, v, kw, torch.randn((len(lens), H, D, Dv), generator=g).cuda()


@pytest.mark.parametrize("bonus", [False, True])
@pytest.mark.parametrize("seg", [16, 48, 96])
@pytest.mark.parametrize("D,Dv", [(1, 1), (16, 31), (64, 33), (65, 96), (128, 130)])
def test_edges_of_chunks_and_segments(ops, monkeypatch, D, Dv, seg, bonus):
    lens, H = [1, 15, 16, 17, 47, 48, 49, 0, 95, 97, 200], 2
    q, k, v, kw, start = _step(lens, H, D, Dv)
    if bonus:
        kw["bonus"] = torch.randn(H * D, device="cuda")
    monkeypatch.setattr(ops, "_scan_segment", lambda *args: seg)
    state = start.clone()
    got = ops.decayed_state_scan(q, k, v, state=state, **kw)
    a = torch.sigmoid(kw["decay_logits"].double()) ** 0.25
    qd, kd, vd = q.double() * 0.25, k.double(), v.double()
    u = kw["bonus"].double().view(H, D, 1) if bonus else None
    want, t = [], 0
    final = start.double()
    for b, n in enumerate(lens):
        S = final[b]
        for t in range(t, t + n):
            kv = kd[t, :, :, None] * vd[t, :, None, :]
            new = a[t, :, :, None] * S + kv
            want.append(((S + u * kv if bonus else new) * qd[t, :, :, None]).sum(1))
            S = new
        t += n > 0
        final[b] = S
    want = torch.stack(want)
    # float32 sums of up to a few hundred addends, decays from float32 exponentials
    assert float((got - want).abs().max()) <= 3e-5 * max(1.0, float(want.abs().max()))
    assert float((state - final).abs().max()) <= 3e-5 * max(1.0, float(final.abs().max()))


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_with_their_column_and_later_tokens(ops, bad):
    q, k, v, kw, start = _step([300, 40], 2, 64, 64)
    clean_state, state = start.clone(), start.clone()
    clean = ops.decayed_state_scan(q, k, v, state=clean_state, **kw)
    v[200, 1, 35] = bad
    got = ops.decayed_state_scan(q, k, v, state=state, **kw)
    hit = torch.zeros_like(clean, dtype=torch.bool)
    hit[200:300, 1, 35] = True
    assert not torch.isfinite(got[hit]).any()
    # (tokens before it in its chunk are summed in another order)
    assert float((got - clean)[~hit].abs().max()) <= 3e-5 * float(clean.abs().max())
    assert not torch.isfinite(state[0, 1, :, 35]).any()
    state[0, 1, :, 35] = clean_state[0, 1, :, 35]
    assert torch.equal(state, clean_state)


@pytest.mark.parametrize("host", [True, False])
@pytest.mark.parametrize("D,Dv,windows", [(64, 33, 3), (128, 130, 6)])
def test_steps_whose_scratch_is_too_large_run_in_windows(ops, monkeypatch, D, Dv, windows, host):
    """Several launches over tokens one after another, whose boundaries fall into sequences, against one launch over all."""
    from qwen3_runtime_b200.ops import cuda

    lens, H, seg = [1, 15, 300, 0, 17, 1, 1, 640, 33, 0, 96], 3, 48
    q, k, v, kw, start = _step(lens, H, D, Dv)
    if not host:
        kw["host_cu_seqlens"] = None
    monkeypatch.setattr(ops, "_scan_segment", lambda *args: seg)
    launched, call = [], ops._call

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    monkeypatch.setattr(ops, "_call", spy)
    out, states = [], []
    for whole in (True, False):
        if not whole:
            most = cuda._scan_scratch(sum(lens), len(lens), H, D, Dv, -(-sum(lens) // seg) + len(lens), True)
            monkeypatch.setattr(cuda, "SCAN_SCRATCH", most // windows + (0 if host else most // 3))
        states.append(start.clone())
        out.append(ops.decayed_state_scan(q, k, v, state=states[-1], **kw))
    assert launched[0] == launched[-1] == "q3_decayed_segment_scan" and len(launched) > 2
    # the sums over a sequence's segments in another order
    assert float((out[0] - out[1]).abs().max()) <= 3e-5 * float(out[0].abs().max())
    assert float((states[0] - states[1]).abs().max()) <= 3e-5 * float(states[0].abs().max())


def test_a_scan_that_is_refused_its_scratch_runs_token_by_token(ops, monkeypatch):
    from qwen3_runtime_b200.ops import cuda

    q, k, v, kw, start = _step([300, 40], 2, 64, 64)
    launched, call = [], ops._call

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    monkeypatch.setattr(ops, "_call", spy)
    monkeypatch.setattr(ops, "_scan_segment", lambda *args: 64)
    want = ops.decayed_state_scan(q, k, v, state=start.clone(), **kw)
    monkeypatch.setattr(cuda, "SCAN_SCRATCH", 1 << 50)
    monkeypatch.setattr(cuda, "_scan_scratch", lambda *args: 1 << 45)  # floats: more than any device has
    got = ops.decayed_state_scan(q, k, v, state=start.clone(), **kw)
    assert launched == ["q3_decayed_segment_scan", "q3_decayed_state_scan"]
    assert float((got - want).abs().max()) <= 3e-5 * float(want.abs().max())
