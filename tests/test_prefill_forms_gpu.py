"""The forms of the tcgen05 prompt kernel beside plain heads (csrc/attention_prefill_tc.cu): both maps of differential
attention as its two row blocks, and attention through a latent on expanded keys and values; against the other kernels of
the same parts, over group sizes, page sizes, masks, portions behind a context, one-token portions and ragged ends."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _layer(ops, spec, page, slots, pages, seed):
    """A mixer with random tensors, and what it needs for steps of its own."""
    from qwen3_runtime_b200.cache.layout import CacheLayout
    from qwen3_runtime_b200.cache.manager import CacheManager
    from qwen3_runtime_b200.cache.storage import CacheStorage
    from qwen3_runtime_b200.engine.batch import BatchBuilder
    from qwen3_runtime_b200.parts.base import BuildContext, build_part

    part = build_part("mixer", spec, BuildContext(dtype=torch.bfloat16, device=torch.device(DEV), ops=ops))
    g = torch.Generator().manual_seed(seed)
    tensors = {}
    for name, ps in part.param_specs().items():
        t = torch.randn(ps.shape, generator=g)
        if ps.kind == "vector":
            t = 0.1 * t if name[:2] in ("lq", "lk") else 1.0 + 0.1 * t
            tensors[name] = t.cuda()
        else:
            tensors[name] = (t * ps.shape[-1] ** -0.5).bfloat16().cuda()
    part.load(tensors)
    layout = CacheLayout({0: part.cache_spec()})
    cache = CacheManager(layout.group_specs, page, pages, slots)
    storage = CacheStorage(layout, page, cache.num_pages, slots, torch.bfloat16, DEV)
    return part, cache, storage, BatchBuilder(cache, DEV, vocab_size=10, max_positions=1 << 20)


def _steps(ops, spec, page, portions, variants, seed=0):
    """Runs ``portions`` (a list of steps, each a list of tokens per request; 0: the request sits the step out) once per
    variant (a function that prepares ``ops``); pages that nothing was written to hold NaN.  The variants' outputs."""
    from qwen3_runtime_b200.engine.batch import StepEntry

    results = []
    for prepare in variants:
        total = [sum(s[i] for s in portions) for i in range(len(portions[0]))]
        part, cache, storage, builder = _layer(ops, spec, page, len(total), sum(-(-n // page) for n in total) + 3, seed)
        for t in storage.tensors:
            for x in t if isinstance(t, tuple) else (t,):
                x.fill_(float("nan"))
        handles = [cache.open(i) for i in range(len(total))]
        g = torch.Generator().manual_seed(seed + 1)
        out = []
        for step_tokens in portions:
            entries = []
            for rc, n in zip(handles, step_tokens):
                if n:
                    cache.reserve(rc, n)
                    entries.append(StepEntry(rc, [0] * n, []))
            step = builder.build(entries, scratch_page=storage.scratch_page, scratch_slot=storage.scratch_slot)
            h = torch.randn((step.num_tokens, int(spec["hidden_size"])), generator=g).bfloat16().cuda()
            restore = prepare(ops)
            try:
                out.append(part.forward(h, step, storage.view(0)).float())
            finally:
                restore()
            ops.raise_if_kernel_error()
            for e in entries:
                cache.commit(e.cache, len(e.tokens))
        results.append(out)
    return results


def _set(**values):
    def prepare(ops):
        before = {k: getattr(ops, k) for k in values}
        for k, v in values.items():
            setattr(ops, k, v)

        def restore():
            for k, v in before.items():
                setattr(ops, k, v)

        return restore

    return prepare


def _close(got, want, factor):
    for a, b in zip(got, want):
        assert bool(torch.isfinite(a).all())
        # factor roundings of bfloat16 (2^-9 of the value) that the two ways do not share, on the output's largest value
        assert float((a - b).abs().max()) <= factor * 2.0 ** -9 * float(b.abs().max())
        assert float((a - b).norm()) <= 0.5 * factor * 2.0 ** -9 * float(b.norm())


RAGGED = [[3, 200, 0, 1, 65], [129, 1, 300, 70, 64], [1, 31, 33, 256, 2]]


@pytest.mark.parametrize("heads,kv_heads,page", [(4, 4, 16), (4, 2, 8), (8, 2, 32), (16, 2, 64), (16, 1, 16)])
@pytest.mark.parametrize("mask", [dict(), dict(chunk=100), dict(chunk=64), dict(window=1), dict(window=90)])
def test_both_maps_as_row_blocks(ops, heads, kv_heads, page, mask):
    from qwen3_runtime_b200.config import PartSpec

    spec = PartSpec("differential_attention", dict(hidden_size=128, num_heads=heads, num_kv_heads=kv_heads, dim=64, vdim=128,
                                                   scale=0.3, diff=0.4, eps=1e-5, **mask))
    launched = []
    call = ops._call

    def spy(group, name, what, *args):
        launched.append(name)
        return call(group, name, what, *args)

    ops._call = spy
    try:
        got, want = _steps(ops, spec, page, RAGGED, [_set(), _set(differential_tc=False)])
    finally:
        del ops._call
    assert launched.count("q3_diff_attention_prefill_tc") == len(RAGGED) and "q3_paged_attention_diff" in launched
    # probabilities are rounded to bfloat16 here and not in the general kernel, and the subtraction of the two maps lifts
    # that rounding by up to (1 + lambda) / |1 - lambda| (about 4 for lambda near 0.4 .. 0.6)
    _close(got, want, 12)


@pytest.mark.parametrize("heads,kv_heads,mask", [(4, 2, dict(chunk=100)), (16, 2, dict(window=90)), (4, 4, dict())])
def test_the_mma_sync_kernel_at_the_same_sizes(ops, heads, kv_heads, mask):
    """It takes the steps whose longest sequence fills no block of 128 rows."""
    from qwen3_runtime_b200.config import PartSpec

    spec = PartSpec("differential_attention", dict(hidden_size=128, num_heads=heads, num_kv_heads=kv_heads, dim=64, vdim=128,
                                                   scale=0.3, diff=0.4, eps=1e-5, **mask))
    for portions in (RAGGED, [[2, 3, 0, 1, 7], [1, 2, 3, 0, 0]]):
        got, want = _steps(ops, spec, 16, portions, [_set(differential_tcgen05=False), _set(differential_tc=False)])
        _close(got, want, 12)


@pytest.mark.parametrize("heads,q_rank,gate,pairing,page", [(2, 64, None, "interleaved", 16), (3, 0, "sigmoid", "half", 8),
                                                          (16, 96, None, "interleaved", 64)])
@pytest.mark.parametrize("window", [None, 1, 64, 90, 300])
@pytest.mark.parametrize("kv_rank", [64, 512])
def test_expanded_keys_and_values(ops, heads, q_rank, gate, pairing, page, window, kv_rank):
    from qwen3_runtime_b200.config import PartSpec

    position = (PartSpec("rope_interleaved", dict(rotary_dim=64, theta=1e4)) if pairing == "interleaved" else
                PartSpec("rotary_scaled", dict(rotary_dim=64, theta=1e4, pairing="half",
                                               scaling=dict(kind="ramp", factor=8.0, original=512.0, fast=32.0, slow=1.0))))
    spec = PartSpec("latent_attention", dict(hidden_size=128, num_heads=heads, dim=128, rot_dim=64, vdim=128, q_rank=q_rank,
                                             kv_rank=kv_rank, eps=1e-5, scale=192 ** -0.5, window=window, sink=True, gate=gate,
                                             position=position))
    launched = []
    call = ops._call

    def spied(**values):
        def prepare(ops):
            launched.append([])
            ops._call = lambda group, name, what, *args: (launched[-1].append(name), call(group, name, what, *args))[1]
            undo = _set(**values)(ops)

            def restore():
                undo()
                del ops._call

            return restore

        return prepare

    got, want = _steps(ops, spec, page, RAGGED, [spied(LATENT_EXPAND_PAIRS=0), spied(latent_expand=False)])
    for step, names in enumerate(launched):  # every step of the first variant expands, none of the second
        expanded = step < len(RAGGED)
        assert names.count("q3_latent_gather") == names.count("q3_dense_attention_prefill_tc") == int(expanded)
        assert any(n in names for n in ("q3_latent_attention", "q3_latent_attention_tc")) != expanded
    # queries, keys, values and the attended rows are rounded to bfloat16 at other places: four roundings on each side
    _close(got, want, 12)


@pytest.mark.parametrize("window", [None, 90])
@pytest.mark.parametrize("expand", [True, False])
def test_latent_attention_against_float64(ops, window, expand):
    """Both ways beside the layer as it is defined, in float64 on the layer's own bfloat16 tensors and rows."""
    from qwen3_runtime_b200.config import PartSpec
    from qwen3_runtime_b200.engine.batch import StepEntry

    H, rank, W = 3, 64, 128
    spec = PartSpec("latent_attention", dict(hidden_size=W, num_heads=H, dim=128, rot_dim=64, vdim=128, q_rank=0, kv_rank=rank,
                                             eps=1e-5, scale=192 ** -0.5, window=window, sink=True, gate=None,
                                             position=PartSpec("rope_interleaved", dict(rotary_dim=64, theta=1e4))))
    part, cache, storage, builder = _layer(ops, spec, 16, 3, 60, 3)
    g = torch.Generator().manual_seed(3)  # the tensors that _layer drew
    t = {}
    for name, ps in part.param_specs().items():
        x = torch.randn(ps.shape, generator=g)
        t[name] = ((1.0 + 0.1 * x) if ps.kind == "vector" else (x * ps.shape[-1] ** -0.5).bfloat16()).double()
    handles = [cache.open(i) for i in range(3)]
    past = [torch.zeros((0, rank + 64), dtype=torch.float64) for _ in handles]
    inv = (1e4 ** (-torch.arange(0, 64, 2).float() / 64)).double()

    def turn(x, pos):  # interleaved pairs
        a = pos.double()[:, None] * inv
        c, s = (f(a).reshape(-1, *[1] * (x.dim() - 2), 32) for f in (torch.cos, torch.sin))
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, u * s + v * c], -1).flatten(-2)

    for lens in ([5, 200, 64], [130, 1, 70]):
        entries = []
        for rc, n in zip(handles, lens):
            cache.reserve(rc, n)
            entries.append(StepEntry(rc, [0] * n, []))
        step = builder.build(entries, scratch_page=storage.scratch_page, scratch_slot=storage.scratch_slot)
        h = torch.randn((sum(lens), W), generator=g).bfloat16()
        restore = (_set(LATENT_EXPAND_PAIRS=0) if expand else _set(latent_expand=False))(ops)
        try:
            out = part.forward(h.cuda(), step, storage.view(0)).cpu().double()
        finally:
            restore()
        ops.raise_if_kernel_error()
        at = 0
        for b, n in enumerate(lens):
            x = h[at:at + n].double()
            pos = torch.arange(past[b].shape[0], past[b].shape[0] + n)
            q = (x @ t["q"].T).view(n, H, 192)
            q = torch.cat([q[..., :128], turn(q[..., 128:], pos)], -1)
            c = x @ t["dkv"].T
            row = torch.cat([c[:, :rank] / (c[:, :rank].pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * t["dkv.norm"],
                             turn(c[:, rank:], pos)], -1)
            past[b] = torch.cat([past[b], row])
            k = torch.cat([(past[b][:, :rank] @ t["uk"].T).view(-1, H, 128), past[b][:, None, rank:].expand(-1, H, -1)], -1)
            v = (past[b][:, :rank] @ t["uv"].T).view(-1, H, 128)
            s = torch.einsum("qhd,khd->hqk", q, k) * 192 ** -0.5
            key = torch.arange(past[b].shape[0])
            hidden = key[None] > pos[:, None]
            if window:
                hidden |= key[None] <= pos[:, None] - window
            s = s.masked_fill(hidden, float("-inf"))
            p = torch.softmax(torch.cat([s, t["sink"].view(H, 1, 1).expand(H, n, 1)], -1), -1)[..., :-1]
            want = torch.einsum("hqk,khd->qhd", p, v).reshape(n, -1) @ t["o"].T
            got = out[at:at + n]
            # five roundings to bfloat16 (2^-9 each) on the way: row, query, key and value, attended row, output
            assert float((got - want).norm()) <= 5 * 2.0 ** -9 * 2 * float(want.norm()), (b, n)
            at += n
        for e in entries:
            cache.commit(e.cache, len(e.tokens))


def test_which_steps_expand(ops):
    from types import SimpleNamespace

    def rows(spans, window, **kw):
        cu = [0]
        for _c, n in spans:
            cu.append(cu[-1] + n)
        step = SimpleNamespace(decode_only=kw.get("decode", False), captured_width=0, host_cu_seqlens=cu,
                               host_kv_lens=[c + n for c, n in spans])
        return ops.latent_expand_rows(step, heads=3, dim=128, rot_dim=64, value_dim=128, kv_rank=512, window=window,
                                      dtype=torch.bfloat16)

    assert rows([(0, 2048)], None) == 2048 and rows([(0, 63)], None) == 63 and rows([(0, 62)], None) == 0
    assert rows([(8000, 8)], None) == 0 and rows([(8000, 8)], 1024) == 0
    assert rows([(1000, 512)], 100) == 512 + 1000 - 901 // 64 * 64
    assert rows([(5, 1), (9, 1)], None, decode=True) == 0


def test_a_step_without_room_for_expanded_rows_stays_in_the_latent_space(ops):
    from qwen3_runtime_b200.config import PartSpec

    spec = PartSpec("latent_attention", dict(hidden_size=128, num_heads=32, dim=128, rot_dim=64, vdim=128, q_rank=64, kv_rank=64,
                                             eps=1e-5, scale=192 ** -0.5, window=None, sink=True, gate=None,
                                             position=PartSpec("rope_interleaved", dict(rotary_dim=64, theta=1e4))))
    asked = []

    def no_room(ops):
        def expanded(*args, **kw):
            asked.append(kw["page_size"])
            raise torch.OutOfMemoryError("no room for the expanded rows")

        ops.latent_attention_expanded = expanded
        return lambda: ops.__dict__.pop("latent_attention_expanded")

    got, want = _steps(ops, spec, 16, [[300, 64], [100, 0]], [no_room, _set(latent_expand=False)])
    assert asked == [16, 16] and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("pairing,pairs", [("interleaved", 32), ("interleaved", 5), ("half", 32), ("half", 7), ("half", 0)])
def test_queries_turned_beside_the_gathered_rows(ops, pairing, pairs):
    """One launch turns the queries' last 64 columns as rotate_heads does and lays the sequences' cached rows side by side."""
    T, H, width, page, seqs = 37, 3, 40, 8, 2
    g = torch.Generator(device="cuda").manual_seed(pairs)
    q = torch.randn((T, H, 192), generator=g, device="cuda").to(torch.bfloat16)
    positions = torch.randint(0, 5000, (T,), generator=g, device="cuda", dtype=torch.int32)
    freqs = torch.rand(pairs, generator=g, device="cuda") if pairs else None
    pages = torch.randn((9, page, width), generator=g, device="cuda").to(torch.bfloat16)
    table = torch.tensor([[3, 0, 8, -1], [5, 1, 2, 7]], dtype=torch.int32, device="cuda")
    kv, cu = torch.tensor([20, 25], dtype=torch.int32, device="cuda"), torch.tensor([0, 12, 37], dtype=torch.int32, device="cuda")
    rows, base = torch.zeros((45, width), dtype=torch.bfloat16, device="cuda"), torch.zeros(seqs, dtype=torch.int32, device="cuda")
    got, want = torch.zeros((T, H, 64), dtype=torch.bfloat16, device="cuda"), torch.zeros((T, H, 64), dtype=torch.bfloat16, device="cuda")
    ops._call("latent_attention", "q3_latent_gather", "latent_gather", pages.data_ptr(), width, table.data_ptr(), 4, kv.data_ptr(),
              cu.data_ptr(), seqs, page, 0, rows.data_ptr(), base.data_ptr(), 45, q.data_ptr() + 256, q.stride(0), q.stride(1),
              got.data_ptr(), positions.data_ptr(), freqs.data_ptr() if pairs else None, pairs, H, T, ops.PAIRINGS[pairing], 1.25)
    ops.rotate_heads(q[:, :, 128:], want, positions=positions, inv_freq=freqs, pairing=pairing, magnitude=1.25)
    # the same angles and products; a fused multiply-add may stand at another product, then one rounding to bfloat16 moves
    assert float((got.float() - want.float()).abs().max()) <= 2.0 ** -8 * float(want.float().abs().max())
    assert torch.equal(got[:, :, 2 * pairs:], want[:, :, 2 * pairs:])
    at = torch.cat([pages[[3, 0, 8]].flatten(0, 1)[:20], pages[[5, 1, 2, 7]].flatten(0, 1)[:25]])
    assert torch.equal(rows, at) and base.tolist() == [0, 20]
