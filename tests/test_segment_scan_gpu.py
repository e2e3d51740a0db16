"""The decayed state scan in segments (csrc/linear_state.cu) against float64 and against the scan token by token: every form
of decay, rotation, the column of ones and the bonus; sequences of one token, of a segment more or less one, of several
segments, behind an earlier portion; key and value sizes that fill no tile."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

LENS = [[1, 31, 32, 33, 200], [160, 1, 97, 64, 5]]  # two portions of five sequences


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _plain(q, k, v, a, u, S):
    out = []
    for t in range(q.shape[0]):
        kv = k[t, :, :, None] * v[t, :, None, :]
        new = S * a[t, :, :, None] + kv
        read = new if u is None else S + u[:, :, None] * kv
        out.append((q[t, :, :, None] * read).sum(1))
        S = new
    return torch.stack(out), S


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,Dv", [(8, 5), (40, 100), (64, 128), (72, 16), (128, 200)])
@pytest.mark.parametrize("form", ["logits", "double exponential", "head", "head turned", "token ones", "bonus"])
def test_segments_against_float64_and_the_chain(ops, dtype, D, Dv, form):
    g = torch.Generator().manual_seed(D + Dv)
    H, B = 3, len(LENS[0])
    ones = form == "token ones"
    slots = torch.tensor([4, 0, 2, 1, 5], dtype=torch.int32)
    start = torch.randn((6, H, D, Dv + ones), generator=g)
    state = {True: start.clone().cuda(), False: start.clone().cuda()}
    S = [start[s].double() for s in slots.tolist()]
    bias, u = torch.randn(H * D, generator=g), torch.randn(H * D, generator=g)
    inv = 50.0 ** (-torch.arange(D // 4).float() * 4 / D)
    at = [0] * B
    for lens in LENS:
        T = sum(lens)
        cu = torch.tensor([0] + lens).cumsum(0).int()
        pos = torch.cat([torch.arange(a, a + n) for a, n in zip(at, lens)]).int()
        q, k, z = (torch.randn((T, H, D), generator=g).to(dtype) for _ in range(3))
        v = torch.randn((T, H, Dv), generator=g).to(dtype)
        tok_a, tok_k = torch.rand((T, H), generator=g), torch.rand((T, H), generator=g)
        head_a = torch.tensor([0.9, 0.999, 0.2])
        kw = dict(cu_seqlens=cu.cuda(), state_slots=slots.cuda(), num_seqs=B, q_scale=0.5)
        qd, kd, vd = q.double() * 0.5, k.double(), v.double()
        bonus = None
        if form == "logits":
            kw.update(decay_logits=z.cuda(), decay_bias=bias.cuda(), tau=3.0)
            a = torch.sigmoid(z.double() + bias.double().view(H, D)) ** (1 / 3.0)
        elif form == "double exponential" or form == "bonus":
            kw.update(decay_logits=z.cuda(), decay_bias=bias.cuda(), decay_mode="exp_neg_exp")
            a = torch.exp(-torch.exp(z.double() + bias.double().view(H, D)))
            if form == "bonus":
                kw.update(bonus=u.cuda())
                bonus = u.double().view(H, D)
        elif form == "token ones":
            kw.update(token_decay=tok_a.cuda(), token_k_scale=tok_k.cuda(), ones_column=True)
            a = tok_a.double()[:, :, None].expand(T, H, D)
            kd = kd * tok_k.double()[:, :, None]
            vd = torch.cat([vd, torch.ones((T, H, 1), dtype=torch.float64)], dim=2)
        else:
            kw.update(head_decay=head_a.cuda())
            a = head_a.double()[None, :, None].expand(T, H, D)
            if form == "head turned":
                kw.update(inv_freq=inv.cuda(), positions=pos.cuda())
                ang = (pos[:, None].float() * inv).double()[:, None, :]
                c, s, n = ang.cos(), ang.sin(), inv.numel()
                qd, kd = (torch.cat([x[..., :n] * c - x[..., n:2 * n] * s, x[..., n:2 * n] * c + x[..., :n] * s, x[..., 2 * n:]], -1)
                          for x in (qd, kd))
        want = []
        for b, n in enumerate(lens):
            r = slice(int(cu[b]), int(cu[b + 1]))
            o, S[b] = _plain(qd[r], kd[r], vd[r], a[r], bonus, S[b])
            want.append(o)
        want = torch.cat(want)
        got = {}
        for segments in (True, False):
            ops.scan_segments = segments
            assert (ops._scan_segment(T, B, H, D, Dv + ones) > 0) == segments
            got[segments] = ops.decayed_state_scan(q.cuda(), k.cuda(), v.cuda(), state=state[segments], **kw).cpu().double()
        ops.scan_segments = True
        assert dtype == torch.bfloat16 or torch.equal(got[True], got[False])  # float32 stays token by token
        at = [x + n for x, n in zip(at, lens)]
        # float32 sums of up to a few hundred addends (and float32 exponentials) against float64
        bound = 3e-5 * max(1.0, float(want.abs().max()))
        assert float((got[False] - want).abs().max()) <= bound
        assert float((got[True] - want).abs().max()) <= bound
        final = torch.stack(S)
        for segments in (True, False):
            have = state[segments].cpu().double()[slots.long()]
            assert float((have - final).abs().max()) <= 3e-5 * max(1.0, float(final.abs().max()))
            assert torch.equal(state[segments][3].cpu(), start[3]), "a slot of another request was touched"


MIXED = [[1] * 20 + [300] + [1] * 20 + [0, 45, 33], [1] * 40 + [129, 0, 200, 64], [64] * 44, [16] * 44]


@pytest.mark.parametrize("D,Dv", [(64, 128), (128, 72)])
@pytest.mark.parametrize("seg", [None, 32, 48, 300])
def test_steps_of_many_sequences(ops, D, Dv, seg):
    """One-token sequences, empty ones and prompts in one step, more sequences than a warp looks at together; with the
    segment length that the lengths give and with others."""
    g = torch.Generator().manual_seed(D)
    H, B = 5, len(MIXED[0])
    slots = torch.randperm(B + 3, generator=g)[:B].int()
    start = torch.randn((B + 3, H, D, Dv), generator=g)
    state, chain = start.clone().cuda(), start.clone().cuda()
    for lens in MIXED:
        T = sum(lens)
        cu = torch.tensor([0] + lens).cumsum(0)
        q, k, z = (torch.randn((T, H, D), generator=g).bfloat16().cuda() for _ in range(3))
        v = torch.randn((T, H, Dv), generator=g).bfloat16().cuda()
        kw = dict(cu_seqlens=cu.int().cuda(), state_slots=slots.cuda(), num_seqs=B, q_scale=0.5, decay_logits=z,
                  decay_bias=torch.zeros(H * D).cuda(), tau=3.0, host_cu_seqlens=cu.tolist())
        ops.scan_segments = False
        want = ops.decayed_state_scan(q, k, v, state=chain, **kw)
        ops.scan_segments = True
        if seg:
            ops._scan_segment = lambda *args: seg
        try:
            got = ops.decayed_state_scan(q, k, v, state=state, **kw)
        finally:
            ops.__dict__.pop("_scan_segment", None)
        # float32 sums of a few hundred addends in another order
        assert float((got - want).abs().max()) <= 3e-5 * max(1.0, float(want.abs().max()))
        assert float((state - chain).abs().max()) <= 3e-5 * max(1.0, float(chain.abs().max()))
    untouched = [s for s in range(B + 3) if s not in slots.tolist()]
    assert torch.equal(state[untouched].cpu(), start[untouched])


def test_a_scan_without_room_for_its_scratch_runs_token_by_token(ops, monkeypatch):
    from qwen3_runtime_b200.ops import cuda

    H, D, Dv, T = 16, 64, 128, 1024
    q, k, z = (torch.randn((T, H, D), device="cuda").bfloat16() for _ in range(3))
    v = torch.randn((T, H, Dv), device="cuda").bfloat16()
    kw = dict(cu_seqlens=torch.tensor([0, T], dtype=torch.int32, device="cuda"), num_seqs=1, decay_logits=z, tau=3.0,
              state_slots=torch.zeros(1, dtype=torch.int32, device="cuda"), host_cu_seqlens=[0, T])
    launched = []
    call = ops._call

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    monkeypatch.setattr(ops, "_call", spy)
    out = []
    for room in (True, False):
        if not room:  # 2^45 floats: more than any device has
            monkeypatch.setattr(ops, "_scan_segment", lambda *args: 64)
            monkeypatch.setattr(cuda, "_scan_scratch", lambda *args: 1 << 45)
        out.append(ops.decayed_state_scan(q, k, v, state=torch.zeros((1, H, D, Dv), device="cuda"), **kw))
    assert launched == ["q3_decayed_segment_scan", "q3_decayed_state_scan"]
    assert float((out[0] - out[1]).abs().max()) <= 3e-5 * float(out[1].abs().max())
