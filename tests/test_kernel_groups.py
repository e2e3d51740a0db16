"""What a model is going to launch is compiled when it is made: no step waits for a compiler."""

from __future__ import annotations

import inspect
import re

import pytest
import torch

from qwen3_runtime_b200 import Qwen3Config
from qwen3_runtime_b200.config.registry import architecture_for_config
from qwen3_runtime_b200.ops import build
from qwen3_runtime_b200.ops import cuda
from qwen3_runtime_b200.parts.base import BuildContext, product_groups
from qwen3_runtime_b200.parts.model import DecoderModel

BF16, F32 = torch.bfloat16, torch.float32


def _context(dtype):
    return BuildContext(dtype=dtype, device=torch.device("cpu"), ops=None)


def test_every_group_that_a_product_can_launch_is_named():
    methods = ("_product", "_small_product", "_few_product", "_few_parts", "_stream_parts", "_f32_segments", "gated_linear")
    source = "".join(inspect.getsource(getattr(cuda.CudaOps, name)) for name in methods)
    launched = set(re.findall(r'self\._(?:call|get)\(\s*"(\w+)"', source))
    assert launched == {*product_groups(_context(BF16)), *product_groups(_context(F32))}
    assert launched <= set(build.all_groups())


@pytest.mark.parametrize("dtype", [BF16, F32])
def test_a_model_names_its_products_groups(dtype):
    cfg = Qwen3Config(vocab_size=64, hidden_size=32, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, head_dim=16,
                      intermediate_size=48, rms_norm_eps=1e-6, rope_theta=1e4, max_position_embeddings=64,
                      tie_word_embeddings=False)
    model = DecoderModel(architecture_for_config(cfg).build_spec(cfg), _context(dtype))
    assert set(product_groups(model.ctx)) <= set(model.kernel_groups())
    for block in model.blocks:
        assert set(product_groups(model.ctx)) <= set(block.kernel_groups())


def test_preparing_compiles_what_calls_the_launchers_too(monkeypatch):
    asked = []
    monkeypatch.setattr(build, "compile_group", lambda g, **kw: asked.append(g))
    monkeypatch.setattr(build, "_loaded", {"rope_kv": None})
    monkeypatch.setattr(build, "_ready", set())
    monkeypatch.setattr(build, "_maker", None)
    ops = object.__new__(cuda.CudaOps)  # (no device here)
    ops.prepare(["norm", "rope_kv", "a group of other operations"])
    assert sorted(asked) == ["host_call", "norm"]
    ops.prepare(["norm", "sampling"])  # only what this process has not seen compiled
    assert sorted(asked) == ["host_call", "norm", "sampling"]
    asked.clear()
    monkeypatch.setattr(build, "_ready", set())
    monkeypatch.setattr(build, "_maker", False)  # this process has looked for it: there is none
    ops.prepare(["norm"])
    assert asked == ["norm"]


def test_launchers_are_called_without_it_where_it_does_not_compile(monkeypatch):
    def compile_group(group, **kw):
        if group == "host_call":
            raise build.KernelBuildError("no headers")

    monkeypatch.setattr(build, "compile_group", compile_group)
    monkeypatch.setattr(build, "_loaded", {})
    monkeypatch.setattr(build, "_ready", set())
    monkeypatch.setattr(build, "_maker", None)
    object.__new__(cuda.CudaOps).prepare(["norm"])
    fn = object()
    assert build.native_caller(fn) is fn
