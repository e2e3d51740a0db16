"""Waits that run out: second builds of kernels, under other names and with short limits (about 1 ms for a wait, 10 ms for the wait
on what is still in flight), leave boxes out, so that a stage's barrier is a flag that nothing sets.  The kernel must come back by
itself with its error word set, and the context must stay usable."""

from __future__ import annotations

import ctypes
import math

import pytest
import torch

import test_kernels_gpu as tk

pytestmark = pytest.mark.gpu

DEFINES = ("-DQ3_WAIT_LIMIT_CYCLES=2000000ll", "-DQ3_DRAIN_LIMIT_CYCLES=20000000ll", "-DQ3_TEST_WITHHOLD_A_BOX")


@pytest.fixture(scope="module")
def ops():
    from qwen3_runtime_b200.ops.cuda import CudaOps

    return CudaOps()


def _build(group, name):
    from qwen3_runtime_b200.ops import build
    from qwen3_runtime_b200.ops.cuda import _SIGNATURES

    fn = getattr(ctypes.CDLL(str(build.compile_group(group, variant="_withheld_box", defines=DEFINES))), name)
    fn.argtypes, fn.restype = _SIGNATURES[group][name], ctypes.c_int
    return fn


def _expires(fn, *args):
    """Run fn(..., error word, stream); the error word afterwards."""
    word = torch.zeros(1, dtype=torch.int32, device="cuda")
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    code = fn(*args, word.data_ptr(), torch.cuda.current_stream().cuda_stream)
    stop.record()
    assert code == 0
    torch.cuda.synchronize()  # returns: every wait in the kernel is bounded
    assert start.elapsed_time(stop) < 2000.0
    return int(word.item())


@pytest.mark.parametrize("context,tokens", [(0, 20), (700, 100)])
def test_prompt_attention(ops, context, tokens):
    nq, nkv, ps, lens, qlens = 8, 2, 16, [context + tokens], [tokens]
    pr = tk.attention_problem(nq, nkv, 128, ps, lens, qlens, torch.bfloat16, 11)
    step = tk.step_for(lens, qlens)
    out = torch.zeros((tokens, nq * 128), dtype=torch.bfloat16, device="cuda")
    work = -(-(-(-tokens * nq // nkv // 128)) // 2)
    scale = 1 / math.sqrt(128)
    assert _expires(_build("attention_prefill_tc", "q3_paged_attention_prefill_tc"), pr["q"].data_ptr(), pr["q"].stride(0), tokens,
                    pr["k"].data_ptr(), pr["v"].data_ptr(), pr["k"].numel() // 128, pr["bt"].data_ptr(), pr["bt"].shape[1],
                    step.kv_lens.data_ptr(), step.cu_seqlens.data_ptr(), out.data_ptr(), 1, work, nq, nkv, 128, ps, scale, 0, 0,
                    None, None) == 2
    # the ordinary build of the same kernel gives the right result
    ops.paged_attention(pr["q"], pr["q"].stride(0), num_heads=nq, num_kv_heads=nkv, head_dim=128, k_pages=pr["k"],
                        v_pages=pr["v"], block_table=pr["bt"], token_seq=pr["seq"], positions=pr["pos"], out=out,
                        page_size=ps, scale=scale, window=None, step=step)
    ops.raise_if_kernel_error()
    tk.close(out, tk.run_attention(tk.REF, pr, nq, nkv, 128, ps, torch.bfloat16), torch.bfloat16, "after", bf16_tol=1e-2)


@pytest.mark.parametrize("rows", [1, 33, 300])
def test_float32_product(ops, rows):
    N, K = 19456, 1088
    w = torch.randn((N, K), device="cuda")
    x = torch.randn((rows, K), device="cuda")
    segments = ops._f32_segments(x, w)
    assert segments > 0
    parts = torch.zeros(3 * rows * K, dtype=torch.bfloat16, device="cuda")
    planes = torch.zeros((segments, rows, N), device="cuda")
    out = torch.zeros((rows, N), device="cuda")
    assert _expires(_build("gemm_f32", "q3_gemm_f32_split"), x.data_ptr(), K, w.data_ptr(), K, out.data_ptr(), N, rows, N, K,
                    parts.data_ptr(), planes.data_ptr()) == 2
    # the ordinary build of the same kernel gives the right result
    got, want = ops.linear(x, w).double(), x.double() @ w.double().t()
    ops.raise_if_kernel_error()
    assert float((got - want).norm() / want.norm()) < 1e-6


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("M,N,K", [(1, 1024, 512), (48, 24576, 512), (16, 77000, 192), (128, 40000, 256)])
def test_product_of_few_tokens(ops, mode, M, N, K):
    """What is left out is a pair's last item's: its only one, or one behind finished ones, whose epilogue has been through before."""
    x = torch.randn((M, K), device="cuda").to(torch.bfloat16)
    w = (K ** -0.5 * torch.randn(((2 if mode == 2 else 1) * N, K), device="cuda")).to(torch.bfloat16)
    out = torch.zeros((M, N), dtype=torch.float32 if mode == 1 else torch.bfloat16, device="cuda")
    assert _expires(_build("gemm_few_tokens", "q3_gemm_few_tokens"), mode, x.data_ptr(), K, w.data_ptr(), K, out.data_ptr(), N, 1,
                    M, N, K) == 1
    # the ordinary build of the same kernel gives the right result
    ops._few_product(mode, x, w, out, 1, M, N, K)
    ops.raise_if_kernel_error()
    want = x.double() @ w.double().t()
    if mode == 2:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    assert float((out.double() - want).norm() / want.norm()) < (1e-6 if mode == 1 else 2.0 ** -8)


@pytest.mark.parametrize("unit", [0, 1, 2])
@pytest.mark.parametrize("counts", [[1], [33, 0, 256], [8, 40] * 60, [500] * 30])
def test_product_of_routed_experts(ops, unit, counts):
    """As above, with tiles in which the second group of the epilogue has slots and tiles in which it has none."""
    E, S, N, K = len(counts), sum(counts), 520, 136
    chunks = [-(-n // 256) for n in counts]
    offsets, tiles = (torch.tensor([0, *torch.tensor(n).cumsum(0)], dtype=torch.int32, device="cuda") for n in (counts, chunks))
    x = torch.randn((S, K), device="cuda").to(torch.bfloat16)
    w = (K ** -0.5 * torch.randn((E, (2 if unit == 2 else 1) * N, K), device="cuda")).to(torch.bfloat16)
    out = torch.zeros((S, N), dtype=torch.bfloat16, device="cuda")
    args = (unit, w.data_ptr(), x.data_ptr(), out.data_ptr(), S, E, N, K, offsets.data_ptr(), tiles.data_ptr(), 7.0, 1.0, 0.0)
    assert _expires(_build("experts_tcgen05", "q3_expert_tcgen05"), *args) == 1
    # the ordinary build of the same kernel gives the right result
    ops._call("experts_tcgen05", "q3_expert_tcgen05", "expert_tc", *args, ops._error_word(x.device).data_ptr())
    ops.raise_if_kernel_error()
    want = torch.cat([r.double() @ v.double().t() for r, v in zip(x.split(counts), w)])
    if unit == 1:
        want = want.clamp(min=0) ** 2
    if unit == 2:
        want = torch.nn.functional.silu(want[:, :N].clamp(max=7)) * want[:, N:].clamp(-7, 7)
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -7
