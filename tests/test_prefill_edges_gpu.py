"""The tcgen05 prompt kernel where its tiles change kind: portions and contexts beside multiples of a row block's tokens and of
64 keys (tiles that all rows see as a whole take a shorter way), and scores that grow along the keys, so that rows move their
reference point in most tiles; against the plain statement."""

from __future__ import annotations

import math

import pytest
import torch

import test_kernels_gpu as tk

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


@pytest.mark.parametrize("nq,nkv,ps", [(8, 2, 16), (2, 2, 64), (16, 1, 8)])
@pytest.mark.parametrize("growth", [0.0, 40.0])
def test_tiles_beside_the_diagonal(ops, nq, nkv, ps, growth):
    D, block = 128, 128 * nkv // nq
    pairs = [(0, block), (0, block - 1), (0, 2 * block + 1), (63, block), (64, block), (65, 2 * block), (64 - block % 64, block),
             (320, 64), (319, 65), (257, 3 * block - 1)]
    pairs = [(c, n) for c, n in pairs if n > 0]
    lens, qlens = [c + n for c, n in pairs], [n for _c, n in pairs]
    pr = tk.attention_problem(nq, nkv, D, ps, lens, qlens, torch.bfloat16, 97)
    if growth:  # the scores' spread grows along a sequence
        for b, n in enumerate(lens):
            for j in range(-(-n // ps)):
                pr["k"][int(pr["bt"][b, j])] *= 0.1 + growth * j * ps / n / 8
    out = torch.full((pr["T"], nq * D), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.paged_attention(pr["q"], pr["q"].stride(0), num_heads=nq, num_kv_heads=nkv, head_dim=D, k_pages=pr["k"],
                        v_pages=pr["v"], block_table=pr["bt"], token_seq=pr["seq"], positions=pr["pos"], out=out,
                        page_size=ps, scale=1 / math.sqrt(D), window=None, step=tk.step_for(lens, qlens))
    ops.raise_if_kernel_error()
    assert torch.isfinite(out).all(), "every row is written"
    want = tk.run_attention(tk.REF, pr, nq, nkv, D, ps, torch.bfloat16)
    # probabilities are rounded to bfloat16 (2^-9 each), like the output: four roundings of the largest value
    tk.close(out, want, torch.bfloat16, "tcgen05 prefill", bf16_tol=1e-2)


def _portions(ops, nq, nkv, ps, pairs, seed=97):
    """Portions of (context, tokens) each; a call that runs their attention, its output and its inputs."""
    lens, qlens = [c + n for c, n in pairs], [n for _c, n in pairs]
    pr = tk.attention_problem(nq, nkv, 128, ps, lens, qlens, torch.bfloat16, seed)
    out = torch.full((pr["T"], nq * 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    step = tk.step_for(lens, qlens)
    return lambda: ops.paged_attention(
        pr["q"], pr["q"].stride(0), num_heads=nq, num_kv_heads=nkv, head_dim=128, k_pages=pr["k"], v_pages=pr["v"],
        block_table=pr["bt"], token_seq=pr["seq"], positions=pr["pos"], out=out, page_size=ps, scale=1 / math.sqrt(128),
        window=None, step=step), out, pr


@pytest.mark.parametrize("nq,nkv", [(16, 4), (4, 4)])
def test_rows_of_other_sequences_have_no_say_in_a_last_block(ops, nq, nkv):
    """A portion's last block reads query rows of the next portion: whatever they hold, here NaN, stays out of the results."""
    run, out, pr = _portions(ops, nq, nkv, 16, [(700, 100), (0, 70)])
    pr["q"][100:] = float("nan")
    run()
    ops.raise_if_kernel_error()
    want = tk.run_attention(tk.REF, pr, nq, nkv, 128, 16, torch.bfloat16)
    assert torch.isfinite(out[:100]).all() and not torch.isfinite(out[100:]).any()
    # probabilities are rounded to bfloat16 (2^-9 each), like the output: four roundings of the largest value
    tk.close(out[:100], want[:100], torch.bfloat16, "tcgen05 prefill", bf16_tol=1e-2)


def test_a_last_block_that_is_not_full_is_no_slower_than_a_full_one(ops):
    """500 tokens behind 3000 against 512: the same blocks and tiles, but for rows that are none in the last blocks."""
    times = []
    for tokens in (500, 512):
        run, _out, _pr = _portions(ops, 16, 16, 16, [(3000, tokens)])
        events = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(31)]
        run()
        for start, stop in events:
            start.record()
            run()
            stop.record()
        torch.cuda.synchronize()
        times.append(sorted(a.elapsed_time(b) for a, b in events)[15])
    assert times[0] <= 1.08 * times[1], times
