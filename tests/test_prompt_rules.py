"""The kernel table's host-side rules for steps with prompts (no kernel runs)."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

from qwen3_runtime_b200.ops.cuda import CudaOps


def _table():
    """A kernel table of a B200 whose rules can be asked without a device."""
    ops = object.__new__(CudaOps)
    ops.SM_COUNT = 148
    ops.latent_expand = ops.scan_segments = ops.differential_tc = ops.differential_tcgen05 = True
    return ops


class _Counted(list):
    reads = 0

    def __iter__(self):
        self.reads += 1
        return super().__iter__()


def _step(spans):
    cu = [0]
    for _context, new in spans:
        cu.append(cu[-1] + new)
    return SimpleNamespace(decode_only=False, captured_width=0, host_cu_seqlens=cu, extras={},
                           host_kv_lens=_Counted(c + n for c, n in spans))


@pytest.mark.parametrize("window", [None, 100, 4096])
def test_a_steps_layers_share_what_expanding_would_cost(window):
    """Eager steps wait for the host: one walk over the step's sequences per step and window, not one per layer."""
    ops = _table()
    spans = [(0, 300), (777, 40)] + [(4096, 1)] * 40
    rows = pairs = 0
    for c, n in spans:
        first = max(0, c + 1 - window) // 64 * 64 if window else 0
        rows += c + n - first
        pairs += sum(min(p + 1, window) if window else p + 1 for p in range(c, c + n))
    step = _step(spans)
    kw = dict(dim=128, rot_dim=64, value_dim=128, kv_rank=512, window=window, dtype=torch.bfloat16)
    ops.LATENT_EXPAND_PAIRS = pairs / rows * 0.999
    assert [ops.latent_expand_rows(step, heads=h, **kw) for h in (4, 4, 8, 4)] == [rows] * 4
    ops.LATENT_EXPAND_PAIRS = pairs / rows * 1.001 + 1e-9
    assert ops.latent_expand_rows(step, heads=4, **kw) == 0
    assert step.host_kv_lens.reads == 1
    kw["window"] = 77
    ops.latent_expand_rows(step, heads=4, **kw)
    ops.latent_expand_rows(_step(spans), heads=4, **kw)
    assert step.host_kv_lens.reads == 2


def test_a_latent_layer_keeps_its_value_rows_once():
    from qwen3_runtime_b200.config import PartSpec
    from qwen3_runtime_b200.parts.base import BuildContext, build_part

    spec = PartSpec("latent_attention", dict(hidden_size=64, num_heads=2, dim=128, rot_dim=64, vdim=128, q_rank=32, kv_rank=16,
                                             eps=1e-5, scale=0.1, window=None, sink=False,
                                             position=PartSpec("rope_interleaved", dict(rotary_dim=64, theta=1e4))))
    part = build_part("mixer", spec, BuildContext(dtype=torch.bfloat16, device=torch.device("cpu"), ops=_table()))
    g = torch.Generator().manual_seed(0)
    tensors = {n: torch.randn(s.shape, generator=g).to(torch.float32 if s.kind == "vector" else torch.bfloat16)
               for n, s in part.param_specs().items()}
    part.load(dict(tensors))
    assert torch.equal(part.expand, torch.cat([tensors["uk"], tensors["uv"]]))
    assert torch.equal(part.uv.reshape(-1, 16), tensors["uv"]) and part.uv.is_contiguous()
    assert part.uv.untyped_storage().data_ptr() == part.expand.untyped_storage().data_ptr()


@pytest.mark.parametrize("heads,kv_heads,new,kernel", [
    (16, 4, [2], "mma"), (16, 4, [31], "mma"), (16, 4, [32], "tc"), (16, 4, [2, 500], "tc"), (16, 16, [127, 40], "mma"),
    (16, 16, [128], "tc"), (16, 1, [2, 7], "mma"), (16, 1, [8], "tc")])
def test_which_kernel_differential_prompts_take(heads, kv_heads, new, kernel):
    """A step whose longest sequence fills no block of 128 rows stays on the mma.sync kernel; the two have names of their own."""
    ops = _table()
    ops.timing = None
    ops._error_word = lambda device: None
    launched = []
    ops._call = lambda group, name, what, *args: launched.append((name, what))
    step = _step([(0, n) for n in new])
    step.num_seqs, step.max_kv_len = len(new), max(new)
    step.kv_lens = step.cu_seqlens = torch.zeros(len(new) + 1, dtype=torch.int32)
    T = sum(new)
    pages = torch.zeros((4, kv_heads, 16, 128), dtype=torch.bfloat16)
    ops.differential_attention(
        torch.zeros((T, heads * 128), dtype=torch.bfloat16), heads * 128, num_heads=heads, num_kv_heads=kv_heads, map_dim=64,
        value_dim=128, k_pages=pages, v_pages=pages, block_table=torch.zeros((len(new), 2), dtype=torch.int32),
        token_seq=step.kv_lens, positions=step.kv_lens, out=torch.zeros((T, heads * 128), dtype=torch.bfloat16), page_size=16,
        scale=1.0, lam=0.5, eps=1e-6, out_scale=1.0, chunk=2048, step=step)
    assert launched == [{"tc": ("q3_diff_attention_prefill_tc", "differential_attention_tc"),
                         "mma": ("q3_diff_attention_prefill", "differential_attention_mma")}[kernel]]


def _cu(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return tuple(cu)


def test_state_scans_are_cut_by_the_lengths_of_their_sequences():
    from qwen3_runtime_b200.ops.cuda import decayed_scan_segment

    def seg(lens, heads=16, dim=64, vdim=128):
        return decayed_scan_segment(_cu(lens), heads, dim, vdim, 148)

    # single tokens beside a long prompt do not lengthen its segments
    for heads, most in ((16, 128), (32, 256), (64, 512)):
        for singles in (0, 1, 7, 15, 17, 19, 31, 63, 127):
            assert 32 <= seg([1] * (singles // 2) + [2040] + [1] * (singles - singles // 2), heads) <= most
    # one short prompt, or one beside a few tokens: a chain of few tokens is over before segments are joined
    assert seg([64]) == seg([128]) == seg([1, 64, 1, 1, 1]) == seg([128] + [1] * 8) == seg([1] * 4096) == seg([15] * 64) == 0
    # many short prompts fill the SMs as they are: a segment each
    assert seg([64] * 32) == 64 and seg([128] * 16) == 128 and seg([32] * 64) == 32
    # a few prompts' blocks fill the SMs once
    assert seg([2048]) == 114 and seg([2040], 32) == 227 and seg([2040], 16, 128) == 227 and seg([1024, 1024], 32) == 256
    assert seg([2000] * 4, 64) == 2000
    assert seg([0, 0]) == 0 and seg([0, 700, 0]) == seg([700]) > 0
    # scratch (rows, and the segments' states where sequences are cut) stays within 1 GiB
    assert seg([8000] * 4, 64, 128, 128) == 0 and seg([4000], 64, 128, 128) > 0


def test_segments_that_fill_the_sms_once():
    import random

    from qwen3_runtime_b200.ops.cuda import _one_wave

    rnd = random.Random(0)
    for _ in range(500):
        lens, most = [rnd.randint(32, 3000) for _ in range(rnd.randint(1, 20))], rnd.randint(1, 40)
        seg = _one_wave(lens, most)
        count = lambda seg: sum(-(-n // seg) for n in lens)  # noqa: E731
        assert (seg == 0) == (len(lens) > most)
        assert not seg or (count(seg) <= most and (seg == 32 or count(seg - 1) > most))
    assert _one_wave([], 5) == 0


def test_a_scan_with_unknown_lengths_is_cut_as_one_sequence():
    ops = _table()
    assert ops._scan_segment(2048, 1, 16, 64, 128) == ops._scan_segment(2048, 32, 16, 64, 128) == 114
    assert ops._scan_segment(2048, 300, 16, 64, 128) == ops._scan_segment(63, 1, 16, 64, 128) == 0
    assert ops._scan_segment(2048, 1, 16, 136, 128) == 0


def test_which_grouping_needs_scratch():
    need = CudaOps._group_scratch
    assert need(48, 8) == need(256, 48) == need(1, 1) == 0
    assert need(257, 8) == 257 + 8 and need(16, 49) == 16 + 49 and need(1025, 64) == 1025 + 2 * 64


def test_single_tokens_beside_one_delta_prompt_stay_out_of_its_chunks():
    ops = _table()

    def long(lens, heads=16, vdim=128):
        return ops._delta_long(list(_cu(lens)), len(lens), heads, vdim)

    assert long([2000] + [1] * 4) == long([1] * 10 + [2000] + [1] * 10) == 1 and long([1, 700], 8) == 1
    assert long([1000] + [1] * 40) == 41 and long([2000] + [1] * 4, 32) == 5 and long([1500, 548, 1]) == 3
    assert long([1500, 548]) == 2 and long([2048]) == 1 and ops._delta_long(None, 7, 16, 128) == 7


def test_segments_are_whole_chunks_of_a_measured_length():
    from qwen3_runtime_b200.ops.cuda import SCAN_SCRATCH, _scan_scratch, _segments, chunk_segment

    for lens in ([2048], [2040] + [1] * 31, [256] * 8, [64] * 32, [17] * 100, [1000, 33, 0, 700], [4000] * 4):
        for heads, dim, vdim in ((4, 64, 128), (16, 64, 128), (16, 128, 128), (64, 128, 128)):
            for seg in (32, 114, 2000):
                got = chunk_segment(_cu(lens), heads, dim, vdim, 148, seg)
                assert got == seg or (got % 16 == 0 and 16 <= got < max(lens) + 16)
                count, longest = _segments(_cu(lens), got)
                if got != seg:
                    assert _scan_scratch(sum(lens), len(lens), heads, dim, vdim, count, longest > got) <= SCAN_SCRATCH
    # many blocks need no cut, few heads short segments
    assert chunk_segment(_cu([256] * 8), 16, 64, 128, 148, 128) == 256 and chunk_segment(_cu([64] * 32), 16, 64, 128, 148, 64) == 64
    assert chunk_segment(_cu([2048]), 4, 64, 128, 148, 32) < chunk_segment(_cu([2048]), 16, 64, 128, 148, 114) <= 512


def test_large_steps_are_cut_whatever_their_records_take():
    from qwen3_runtime_b200.ops.cuda import SCAN_SCRATCH, _scan_scratch, _scan_windows, decayed_scan_segment

    for tokens, heads, dim, vdim in ((10500, 64, 128, 128), (10000, 64, 128, 256), (20000, 32, 128, 512), (80000, 16, 64, 128)):
        cu = _cu([tokens])
        seg = -(-decayed_scan_segment(cu, heads, dim, vdim, 148) // 16) * 16
        assert seg > 0 and _scan_scratch(tokens, 1, heads, dim, vdim, -(-tokens // seg), seg < tokens) > SCAN_SCRATCH
        assert len(_scan_windows(cu, heads, dim, vdim, seg)[1]) > 1
    ops = _table()
    assert ops._scan_segment(10000, 1, 64, 128, 128) > 0  # the lengths unknown


def test_windows_cover_a_step_and_fit_their_scratch(monkeypatch):
    import random

    from qwen3_runtime_b200.ops import cuda

    rnd = random.Random(0)
    some = [0, 0]
    for _ in range(400):
        heads, dim, vdim = rnd.choice([1, 4, 16]), rnd.choice([64, 128]), rnd.choice([16, 128, 200])
        lens = [rnd.choice([0, 1, 1, rnd.randint(2, 40), rnd.randint(1, 900)]) for _ in range(rnd.randint(1, 40))]
        cu, T, seg = _cu(lens), sum(lens), 16 * rnd.randint(1, 20)
        record, state = cuda._scan_scratch(0, 1, heads, dim, vdim, 0, False), heads * dim * (vdim + 1)
        monkeypatch.setattr(cuda, "SCAN_SCRATCH", rnd.randint(2 * record + state, 60 * (record + state)))
        got, windows = cuda._scan_windows(cu, heads, dim, vdim, seg)
        assert 16 <= got <= seg and got % 16 == 0
        if T == 0:
            continue
        some[len(windows) > 1] += 1
        assert windows[0][0] == 0 and windows[-1][1] == T
        assert all(a[1] == b[0] for a, b in zip(windows, windows[1:]))
        for lo, hi, first, last, segments, cut in windows:
            inside = [min(max(b, lo), hi) - min(max(a, lo), hi) for a, b in zip(cu, cu[1:])]
            assert sum(inside) == sum(inside[first:last]) == hi - lo > 0
            assert segments == sum(-(-n // got) for n in inside) and cut == any(n > got for n in inside)
            assert cuda._scan_scratch(hi - lo, last - first, heads, dim, vdim, segments, cut) <= cuda.SCAN_SCRATCH
        got, windows = cuda._scan_runs(T, len(lens), heads, dim, vdim, seg)
        assert (got == 0) == (not windows)
        for lo, hi, first, last, segments, cut in windows:
            assert (first, last) == (0, len(lens)) and segments >= sum(
                -(-(min(max(b, lo), hi) - min(max(a, lo), hi)) // got) for a, b in zip(cu, cu[1:]))
            assert cuda._scan_scratch(hi - lo, last, heads, dim, vdim, segments, cut) <= cuda.SCAN_SCRATCH
    assert min(some) > 50


def test_the_length_that_was_handed_in_stays_only_where_no_other_fits():
    from qwen3_runtime_b200.ops.cuda import SCAN_SCRATCH, _scan_scratch, _segments, chunk_segment

    kept = chosen = 0
    for lens in ([2048], [2040] + [1] * 31, [256] * 8, [64] * 32, [17] * 100, [1000, 33, 0, 700], [4000] * 4):
        cu = _cu(lens)
        for heads, dim, vdim in ((4, 64, 128), (16, 64, 128), (16, 128, 128), (64, 128, 128)):
            def fits(seg):
                count, longest = _segments(cu, seg)
                return _scan_scratch(sum(lens), len(lens), heads, dim, vdim, count, longest > seg) <= SCAN_SCRATCH

            for seg in (33, 114, 2001):  # none is a multiple of 16
                lengths = {-(-n // 16) * 16 for n in (32, 64, 96, 128, 192, 256, 512, 1024, seg, max(lens)) if n <= max(lens)}
                got = chunk_segment(cu, heads, dim, vdim, 148, seg)
                if any(fits(n) for n in lengths):
                    chosen += 1
                    assert got in lengths and fits(got), (lens, heads, dim, seg, got)
                else:
                    kept += 1
                    assert got == seg
    assert chosen > 60 and kept > 0
