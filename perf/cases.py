"""What a program that serves models with this package has it do, as cases that can be timed and compared.

Two kinds of entry point are called, both as a program calls them:

* whole steps -- ``ModelRunner.run(entries)`` of a Qwen3 dense model: decode steps behind a filled cache (replayed from a
  captured graph, as the engine runs them) and prompts; the answer is the step's logits;
* single layers -- a part from ``build_part`` with its own tensors, the step from ``BatchBuilder`` and the cache behind
  it: grouped-query attention, attention through a latent, differential attention, gated linear attention, the gated
  delta rule, routed experts and the dense gated feed-forward; the answer is the layer's output and the cache or state
  that it wrote.

Sizes are those of ``bench.py``: the Qwen3 shapes with fewer layers, and the w2048 / w4096 layer sizes of the other
designs.  Weights are N(0, 0.02) (norm weights 1 + N(0, 0.02)), layer inputs N(0, 1) as behind a norm.
"""

import math

import torch

PAGE = 16
EPS = 1e-6
DEV = "cuda"

# width, query heads, key/value heads, feed-forward width, tied output head (heads of 128, vocabulary 151936)
DENSE = {"4b": (2560, 32, 8, 9728, True), "8b": (4096, 32, 8, 12288, False), "32b": (5120, 64, 8, 25600, False)}
VOCAB = 151936
LATENT = {"w2048": dict(width=2048, heads=16, q_rank=768, window=1024), "w4096": dict(width=4096, heads=32, q_rank=1536, window=2048)}
EXPERTS = {"w2048": dict(width=2048, experts=64, top=6, ff=1408, shared=2816), "w4096": dict(width=4096, experts=32, top=4, ff=2048, shared=2048)}
GLA = {"w2048": dict(width=2048, heads=16), "w4096": dict(width=4096, heads=32)}  # keys of 64, values of 128, rank 16
DELTA = {"w2048": dict(width=2048, heads=16, kv_heads=8, rank=64), "w4096": dict(width=4096, heads=32, kv_heads=16, rank=128)}
DIFF = {"w2048": dict(width=2048, heads=16, kv_heads=4), "w4096": dict(width=4096, heads=32, kv_heads=8)}  # maps of 64, values of 128


def listed():
    return [
        # one user reading along: a single request's next token; the least work, where latency counts
        dict(name="decode_one", kind="step", size="4b", layers=8, context="512", new="1"),
        # the package's default benchmark point: eight requests behind 4,096 tokens each
        dict(name="decode_batch", kind="step", size="4b", layers=8, context=",".join(["4096"] * 8), new=",".join(["1"] * 8)),
        # continuous batching: 48 requests of unequal lengths, each with its next token
        dict(name="decode_ragged", kind="step", size="8b", layers=4,
             context=",".join(str(64 + 83 * i) for i in range(48)), new=",".join(["1"] * 48)),
        # a prompt of 2,048 tokens, until its first token's logits
        dict(name="prompt_step", kind="step", size="4b", layers=8, context="0", new="2048"),
        # the attention layer of the largest shape over several prompts at once, one of them a later portion
        dict(name="attention_prompts", kind="attention", size="32b", context="0,0,2048,0", new="2500,701,1024,33"),
        # the 32-bit path, which checks the 16-bit one: a feed-forward over a short prompt
        dict(name="mlp_float32", kind="mlp", size="4b", tokens=300, dtype="float32"),
        # routed experts over a prompt, and for one token of each of eight requests
        dict(name="experts_prompt", kind="experts", size="w2048", unit="clamped", tokens=2048),
        dict(name="experts_decode", kind="experts", size="w2048", unit="clamped", tokens=8),
        # attention through a latent with a window and a sink over a prompt
        dict(name="latent_prompt", kind="latent", size="w2048", new="2048"),
        # gated linear attention over a prompt: a matrix state per head, decays per key channel
        dict(name="linear_prompt", kind="gla", size="w2048", new="2048"),
        # the gated delta rule over two prompts of unequal lengths
        dict(name="delta_prompts", kind="delta", size="w2048", new="1500,548"),
        # differential attention under chunks of 2,048 tokens over a long and a short prompt
        dict(name="differential_prompts", kind="diff", size="w2048", new="2333,419"),
    ]


def _spread(rng, low, high):
    """A whole number in low..high, spread over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _prompts(rng, most, low=17, high=2048):
    """Lengths of one to six prompts, ``most`` tokens in all at most."""
    out, left = [], most
    for _ in range(rng.randint(1, 6)):
        n = min(left, _spread(rng, low, high))
        if n < 1:
            break
        out.append(n)
        left -= n
    return out


def _text(numbers):
    return ",".join(str(n) for n in numbers)


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "attention", "mlp", "experts", "experts", "latent", "gla", "delta", "diff"])
    w = rng.choice(["w2048", "w4096"])
    if kind == "decode":
        size, n = rng.choice(["4b", "8b"]), _spread(rng, 1, 64)
        most = _spread(rng, 128, min(4096, 32768 // n))
        return dict(kind="step", size=size, layers=rng.randint(2, 6), new=_text([1] * n),
                    context=_text(rng.randint(max(1, most // 8), most) for _ in range(n)))
    if kind == "prompt":
        new = _prompts(rng, 2048)
        return dict(kind="step", size=rng.choice(["4b", "8b"]), layers=rng.randint(2, 4), context=_text([0] * len(new)), new=_text(new))
    if kind == "attention":
        new = _prompts(rng, 4096)
        return dict(kind="attention", size=rng.choice(list(DENSE)), context=_text(rng.choice([0, 0, rng.randint(1, 2048)]) for _ in new),
                    new=_text(new))
    if kind == "mlp":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        return dict(kind="mlp", size=rng.choice(["4b", "8b"]), dtype=dtype, tokens=_spread(rng, 1, 300 if dtype == "float32" else 3000))
    if kind == "experts":
        return dict(kind="experts", size=w, unit=rng.choice(["clamped", "relu2"]), tokens=_spread(rng, 1, 2500))
    return dict(kind=kind, size=w, new=_text(_prompts(rng, 2500)))


# ---- sizes and tensors ---------------------------------------------------------------------------------------------


def _numbers(text):
    return [int(x) for x in text.split(",")]


def _dense_shapes(size, layers):
    W, H, G, F, tied = DENSE[size]
    out = {"model.embed_tokens.weight": (VOCAB, W)}
    for i in range(layers):
        p = f"model.layers.{i}."
        out.update({p + "input_layernorm.weight": (W,), p + "post_attention_layernorm.weight": (W,)})
        out.update({p + "self_attn." + n: s for n, s in _attention_shapes(W, H, G).items()})
        out.update({p + "mlp." + n: s for n, s in _mlp_shapes(W, F).items()})
    out["model.norm.weight"] = (W,)
    if not tied:
        out["lm_head.weight"] = (VOCAB, W)
    return out


def _attention_shapes(W, H, G):
    return {"q_proj.weight": (H * 128, W), "k_proj.weight": (G * 128, W), "v_proj.weight": (G * 128, W), "o_proj.weight": (W, H * 128),
            "q_norm.weight": (128,), "k_norm.weight": (128,)}


def _mlp_shapes(W, F):
    return {"gate_proj.weight": (F, W), "up_proj.weight": (F, W), "down_proj.weight": (W, F)}


def _shapes(case):
    """Name -> shape of every tensor of the case's model or layer."""
    kind = case["kind"]
    if kind == "step":
        return _dense_shapes(case["size"], case["layers"])
    if kind in ("attention", "mlp"):
        W, H, G, F, _ = DENSE[case["size"]]
        return _attention_shapes(W, H, G) if kind == "attention" else _mlp_shapes(W, F)
    if kind == "latent":
        z = LATENT[case["size"]]
        W, H, R = z["width"], z["heads"], z["q_rank"]
        return {"dq": (R, W), "dq.norm": (R,), "uq": (H * 192, R), "dkv": (576, W), "dkv.norm": (512,), "uk": (H * 128, 512),
                "uv": (H * 128, 512), "o": (W, H * 128), "sink": (H,)}
    if kind == "gla":
        z = GLA[case["size"]]
        W, H = z["width"], z["heads"]
        return {"q": (H * 64, W), "k": (H * 64, W), "v": (H * 128, W), "g": (H * 128, W), "o": (W, H * 128), "norm": (128,),
                "a1": (16, W), "a2": (H * 64, 16), "a2.b": (H * 64,)}
    if kind == "delta":
        z = DELTA[case["size"]]
        W, H, G, R = z["width"], z["heads"], z["kv_heads"], z["rank"]
        return {"q": (G * 128, W), "q.conv": (G * 128, 4), "k": (G * 128, W), "k.conv": (G * 128, 4), "v": (H * 128, W),
                "v.conv": (H * 128, 4), "b": (H, W), "A_log": (H,), "norm": (128,), "a1": (R, W), "a2": (H * 128, R),
                "dt_bias": (H * 128,), "g1": (R, W), "g2": (H * 128, R), "o": (W, H * 128)}
    if kind == "diff":
        z = DIFF[case["size"]]
        W, H, G = z["width"], z["heads"], z["kv_heads"]
        return {"q": (H * 128, W), "k": (G * 128, W), "v": (G * 128, W), "q.norm": (64,), "k.norm": (64,), "o": (W, H * 128),
                "lq1": (64,), "lk1": (64,), "lq2": (64,), "lk2": (64,)}
    z = EXPERTS[case["size"]]
    W, F, S = z["width"], z["ff"], z["shared"]
    out = {}
    gated = case["unit"] == "clamped"
    for e in range(z["experts"]):
        out.update({f"e{e}.gate": (F, W)} if gated else {})
        out.update({f"e{e}.up": (F, W), f"e{e}.down": (W, F)})
    out["router"] = (z["experts"], W)
    out.update({"shared.gate": (S, W)} if gated else {"shared.sg": (1, W)})
    out.update({"shared.up": (S, W), "shared.down": (W, S)})
    return out


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _weights(case, seed):
    """The stored tensors: matrices in the compute type, vectors, routers and convolutions in 32 bits."""
    g = torch.Generator(device=DEV).manual_seed(2 * int(seed))
    out = {}
    for name, shape in _shapes(case).items():
        t = torch.randn(shape, generator=g, device=DEV, dtype=torch.float32)
        last = name.rsplit(".", 1)[-1]
        if name == "A_log":  # decay rates from 1 to 16
            t = torch.rand(shape, generator=g, device=DEV) * math.log(16.0)
        elif name == "dt_bias":  # steps from about 0.001 to 0.1
            t = -6.9 + 4.7 * torch.rand(shape, generator=g, device=DEV)
        elif last in ("lq1", "lk1", "lq2", "lk2"):
            t = 0.1 * t
        elif last == "conv":
            t = 0.5 * t
        elif len(shape) == 1:
            t = 1.0 + 0.02 * t
        elif name == "router":
            t = 0.02 * t
        else:
            t = (0.02 * t).to(_dtype(case))
        out[name] = t
    return out


def _inputs(case, seed):
    """Token ids (a step), else the layer's input rows; and keys and values of the tokens that are cached already."""
    g = torch.Generator(device=DEV).manual_seed(2 * int(seed) + 1)
    if case["kind"] == "step":
        n = sum(_numbers(case["new"]))
        ids = torch.randint(1, 1000, (n,), generator=torch.Generator().manual_seed(2 * int(seed) + 1)).tolist()
        return ids, _cached(case, g, case["layers"])
    if case["kind"] in ("mlp", "experts"):
        n, W = case["tokens"], (DENSE[case["size"]][0] if case["kind"] == "mlp" else EXPERTS[case["size"]]["width"])
    else:
        n = sum(_numbers(case["new"]))
        W = DENSE[case["size"]][0] if case["kind"] == "attention" else {"latent": LATENT, "gla": GLA, "delta": DELTA,
                                                                          "diff": DIFF}[case["kind"]][case["size"]]["width"]
    h = torch.randn((n, W), generator=g, device=DEV, dtype=torch.float32).to(_dtype(case))
    return h, _cached(case, g, 1) if case["kind"] == "attention" else None


def _cached(case, g, layers):
    """Per request ``[layers, 2, cached tokens, key/value heads, 128]`` in 16 bits, or None."""
    G = DENSE[case["size"]][2]
    return [torch.randn((layers, 2, c, G, 128), generator=g, device=DEV, dtype=torch.bfloat16) if c else None
            for c in _numbers(case["context"])]


# ---- the package -----------------------------------------------------------------------------------------------------


def _fill(view, table, cached):
    """Write a request's cached keys and values ``[2, c, G, 128]`` into the pages of its block table."""
    c = cached.shape[1]
    pages = -(-c // PAGE)
    rows = torch.nn.functional.pad(cached, (0, 0, 0, 0, 0, pages * PAGE - c)).unflatten(1, (pages, PAGE)).transpose(2, 3)
    at = torch.tensor(table[:pages], device=DEV)
    view.k_pages[at], view.v_pages[at] = rows[0], rows[1]


class _Decode:
    """Decode steps of requests that hold ``contexts`` tokens.  They go on token by token; after LAST tokens the requests
    end and others of the same lengths begin, as in a served batch."""

    LAST = 128

    def __init__(self, rt, contexts, ids, cached=None):
        self.rt, self.contexts, self.ids = rt, contexts, ids
        self.handles, self.done = [], 0
        self.start(cached)

    def start(self, cached=None):
        cache = self.rt.cache
        for rc in self.handles:
            cache.close(rc)
        self.handles, self.done = [], 0
        for i, c in enumerate(self.contexts):
            rc = cache.open(i)
            cache.reserve(rc, c)
            if cached is not None and cached[i] is not None:
                for layer in range(cached[i].shape[0]):
                    _fill(self.rt.storage.view(layer), rc.tables[0], cached[i][layer])
            cache.commit(rc, c)
            rc.needs_state_reset = False
            self.handles.append(rc)

    def step(self):
        from qwen3_runtime_b200.engine.batch import StepEntry

        if self.done == self.LAST:
            self.start()
        self.done += 1
        entries = []
        for rc, token in zip(self.handles, self.ids):
            self.rt.cache.reserve(rc, 1)
            entries.append(StepEntry(rc, [token], [0]))
        return self.rt.runner.run(entries)


def _prepare_step(case, seed):
    from qwen3_runtime_b200.config import Qwen3Config
    from qwen3_runtime_b200.engine.factory import build_model, build_runtime
    from qwen3_runtime_b200.weights import DictSource

    W, H, G, F, tied = DENSE[case["size"]]
    cfg = Qwen3Config(vocab_size=VOCAB, hidden_size=W, num_hidden_layers=case["layers"], num_attention_heads=H, num_key_value_heads=G,
                      head_dim=128, intermediate_size=F, rms_norm_eps=EPS, rope_theta=1e6, max_position_embeddings=8192,
                      tie_word_embeddings=tied)
    contexts, new = _numbers(case["context"]), _numbers(case["new"])
    ids, cached = _inputs(case, seed)
    model = build_model(cfg, DictSource(_weights(case, seed)))
    pages = sum(-(-(c + n + _Decode.LAST) // PAGE) for c, n in zip(contexts, new))
    rt = build_runtime(model, block_size=PAGE, num_kv_blocks=pages, max_num_seqs=len(new), cuda_graph=True)
    if max(new) > 1:
        split, at = [], 0
        for n in new:
            split.append(ids[at:at + n])
            at += n
        return dict(case=case, rt=rt, prompts=split)
    decode = _Decode(rt, contexts, ids)
    decode.step()  # a served model has its decode step captured
    decode.start(cached)
    return dict(case=case, decode=decode)


def _part(case):
    """Category and spec of the case's layer."""
    from qwen3_runtime_b200.config import PartSpec

    kind, size = case["kind"], case["size"]
    if kind == "attention":
        W, H, G, _F, _ = DENSE[size]
        return "mixer", PartSpec("paged_attention", dict(
            hidden_size=W, num_heads=H, num_kv_heads=G, head_dim=128, qk_norm_eps=EPS, window=None,
            position=PartSpec("rope_neox", dict(rotary_dim=128, theta=1e6, max_positions=8192))))
    if kind == "mlp":
        W, _H, _G, F, _ = DENSE[size]
        return "feed_forward", PartSpec("gated_mlp", dict(hidden_size=W, intermediate_size=F, activation="silu"))
    if kind == "latent":
        z = LATENT[size]
        return "mixer", PartSpec("latent_attention", dict(
            hidden_size=z["width"], num_heads=z["heads"], dim=128, rot_dim=64, vdim=128, q_rank=z["q_rank"], kv_rank=512, eps=EPS,
            scale=192 ** -0.5, window=z["window"], sink=True,
            position=PartSpec("rope_interleaved", dict(rotary_dim=64, theta=10000.0))))
    if kind == "gla":
        z = GLA[size]
        return "mixer", PartSpec("gla", dict(hidden_size=z["width"], num_heads=z["heads"], dim=64, vdim=128, tau=16.0, eps=EPS,
                                             decay_rank=16))
    if kind == "delta":
        z = DELTA[size]
        return "mixer", PartSpec("gated_delta", dict(
            hidden_size=z["width"], num_heads=z["heads"], num_kv_heads=z["kv_heads"], dim=128, vdim=128, taps=4, decay_rank=z["rank"],
            gate_rank=z["rank"], eps=EPS))
    if kind == "diff":
        z = DIFF[size]
        return "mixer", PartSpec("differential_attention", dict(
            hidden_size=z["width"], num_heads=z["heads"], num_kv_heads=z["kv_heads"], dim=64, vdim=128, scale=64 ** -0.5, diff=0.6,
            eps=EPS, chunk=2048))
    z = EXPERTS[size]
    shared = dict(hidden_size=z["width"], num_experts=z["experts"], top=z["top"], expert_size=z["ff"], shared_size=z["shared"])
    if case["unit"] == "clamped":
        return "feed_forward", PartSpec("routed_experts", dict(
            shared, limit=7.0, alpha=1.702, up_offset=1.0, score="sigmoid", renormalize=False, weight_on="input", shared_limit=7.0))
    return "feed_forward", PartSpec("routed_experts", dict(
        shared, activation="relu2", score="softmax_chosen", weight_on="output", shared_gate="sigmoid"))


def _prepare_layer(case, seed):
    from qwen3_runtime_b200.cache.layout import CacheLayout
    from qwen3_runtime_b200.cache.manager import CacheManager
    from qwen3_runtime_b200.cache.storage import CacheStorage
    from qwen3_runtime_b200.engine.batch import BatchBuilder, StepEntry
    from qwen3_runtime_b200.ops.cuda import CudaOps
    from qwen3_runtime_b200.parts.base import BuildContext, build_part

    category, spec = _part(case)
    ops = CudaOps()
    part = build_part(category, spec, BuildContext(dtype=_dtype(case), device=torch.device(DEV), ops=ops))
    ops.prepare(part.kernel_groups())
    part.load(_weights(case, seed))
    h, cached = _inputs(case, seed)
    if category == "feed_forward":
        return dict(case=case, part=part, h=h)
    new = _numbers(case["new"])
    contexts = _numbers(case["context"]) if cached is not None else [0] * len(new)
    layout = CacheLayout({0: part.cache_spec()})
    cache = CacheManager(layout.group_specs, PAGE, sum(-(-(c + n) // PAGE) for c, n in zip(contexts, new)), len(new))
    storage = CacheStorage(layout, PAGE, cache.num_pages, len(new), _dtype(case), DEV)
    builder = BatchBuilder(cache, DEV, vocab_size=VOCAB, max_positions=1 << 20)
    view, entries = storage.view(0), []
    for i, (c, n) in enumerate(zip(contexts, new)):
        rc = cache.open(i)
        cache.reserve(rc, c)
        if c:
            _fill(view, rc.tables[0], cached[i][0])
        cache.commit(rc, c)
        cache.reserve(rc, n)
        entries.append(StepEntry(rc, [0] * n, []))
    step = builder.build(entries, scratch_page=storage.scratch_page, scratch_slot=storage.scratch_slot)
    return dict(case=case, part=part, h=h, step=step, storage=storage, view=view, builder=builder, slots=[e.cache.slot for e in entries])


def prepare(case, seed):
    return _prepare_step(case, seed) if case["kind"] == "step" else _prepare_layer(case, seed)


def run(state):
    if "decode" in state:
        return state["decode"].step()
    if "prompts" in state:  # new requests come, their prompts run as one step, the last token's logits are wanted
        from qwen3_runtime_b200.engine.batch import StepEntry

        rt, entries = state["rt"], []
        for i, tokens in enumerate(state["prompts"]):
            rc = rt.cache.open(i)
            rt.cache.reserve(rc, len(tokens))
            entries.append(StepEntry(rc, tokens, [len(tokens) - 1]))
        logits = rt.runner.run(entries)
        for e in entries:
            rt.cache.close(e.cache)
        return logits
    kind = state["case"]["kind"]
    if kind in ("mlp", "experts"):
        return state["part"].forward(state["h"], None)
    if kind in ("gla", "delta"):  # a request's state starts from zero
        state["storage"].zero_state_slots(state["slots"])
    step = state["step"]
    step.extras = {}
    view = state["view"]
    out = state["part"].forward(state["h"], step, view)
    n = len(state["slots"])
    if kind == "gla":
        return dict(out=out, state=view.state[:n])
    if kind == "delta":
        return dict(out=out, state=view[0].state[:n], ring=view[1].state[:n])
    if kind == "latent":
        return dict(out=out, pages=view.latent_pages)
    return dict(out=out, keys=view.k_pages, values=view.v_pages)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    e = 4 if case.get("dtype") == "float32" else 2
    sizes = _shapes(case)
    matrices = {n: math.prod(s) for n, s in sizes.items() if len(s) == 2 and not n.endswith(".conv")}
    if kind in ("mlp", "experts"):
        T = case["tokens"]
        if kind == "mlp":
            n, W = sum(matrices.values()), DENSE[case["size"]][0]
            return {"bytes": e * (n + 2 * T * W), "flops": 2.0 * T * n}
        z = EXPERTS[case["size"]]
        one = sum(n for name, n in matrices.items() if name.startswith("e0."))
        rest = sum(n for name, n in matrices.items() if name.startswith("shared"))
        read = min(z["experts"], T * z["top"]) if T * z["top"] < z["experts"] else \
            z["experts"] * (1.0 - (1.0 - z["top"] / z["experts"]) ** T)  # distinct experts, uniformly chosen
        return {"bytes": 2 * (read * one + rest + 2 * T * z["width"]) + 4 * matrices["router"],
                "flops": 2.0 * T * (z["top"] * one + rest + matrices["router"])}
    new = _numbers(case["new"])
    T = sum(new)
    if kind in ("step", "attention"):
        W, H, G, _F, tied = DENSE[case["size"]]
        layers = case.get("layers", 1)
        spans = list(zip(_numbers(case["context"]), new))
        pairs = sum(n * c + n * (n + 1) / 2 for c, n in spans)
        held = sum(c + n for c, n in spans)
        kv = layers * 2 * G * 128 * 2 * (held + (T if kind == "step" and max(new) > 1 else 0))
        body = sum(n for name, n in matrices.items() if "embed" not in name and "lm_head" not in name)
        head = VOCAB * W if kind == "step" else 0
        rows = len(new) if kind == "step" else 0
        return {"bytes": 2 * (body + head) + kv + 2 * T * W * (1 if kind == "step" else 2) + 4 * rows * VOCAB,
                "flops": 2.0 * T * body + 2.0 * rows * head + layers * 4.0 * H * 128 * pairs}
    n = sum(matrices.values())
    z = {"latent": LATENT, "gla": GLA, "delta": DELTA, "diff": DIFF}[kind][case["size"]]
    io, H = 2 * (n + 2 * T * z["width"]), z["heads"]
    if kind == "latent":  # scores over dim + rot_dim and values of 128 per head, as the layer is defined
        pairs = sum(sum(min(i + 1, z["window"]) for i in range(x)) for x in new)
        return {"bytes": io + 2 * T * 576, "flops": 2.0 * T * n + 2.0 * H * (192 + 128) * pairs}
    if kind == "diff":
        pairs = sum((i % 2048) + 1 for x in new for i in range(x))
        return {"bytes": io + 2 * T * z["kv_heads"] * 256, "flops": 2.0 * T * n + 2.0 * H * (128 + 256) * pairs}
    state = H * (64 if kind == "gla" else 128) * 128
    return {"bytes": io + 4 * len(new) * state, "flops": 2.0 * T * n + (6.0 if kind == "gla" else 8.0) * T * state}


def tolerance(case):
    """About four times what sums in another order differ by: a layer's output lies 0.0035 to 0.005 from 64 bits, the logits
    of a model of two to eight layers 0.01 to 0.015, the 32-bit feed-forward 2.2e-6."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.03} if case["kind"] == "step" else {"rel": 0.015}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------


def _rms(x, w=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _turn(x, start, theta, interleaved):
    """Rotate ``x`` ``[n, heads, d]`` of the tokens at ``start ..`` over all of d."""
    n, d = x.shape[0], x.shape[-1]
    f = theta ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float64) / d)
    a = (torch.arange(start, start + n, device=DEV, dtype=torch.float64)[:, None] * f)[:, None, :]
    c, s = a.cos(), a.sin()
    if interleaved:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)
    u, v = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], dim=-1)


def _softmax_sum(q, k, v, start, scale, window=None, chunk=None, sink=None):
    """Causal attention of one head: q ``[n, d]`` at positions ``start ..`` over k, v ``[L, .]`` (rows from position 0)."""
    i = torch.arange(start, start + q.shape[0], device=DEV)[:, None]
    j = torch.arange(k.shape[0], device=DEV)[None, :]
    hidden = j > i
    if window:
        hidden |= j <= i - window
    if chunk:
        hidden |= torch.div(j, chunk, rounding_mode="floor") != torch.div(i, chunk, rounding_mode="floor")
    z = (scale * (q @ k.T)).masked_fill_(hidden, -math.inf)
    if sink is not None:
        z = torch.cat([z, sink.expand(z.shape[0], 1)], dim=1)
    return torch.softmax(z, dim=1)[:, : k.shape[0]] @ v


def _exact_attention(h, w, H, G, spans, cached):
    """Output rows of the grouped-query attention layer; ``cached``: per request ``[2, c, G, 128]`` or None."""
    D, out, at = 128, [], 0
    q, k, v = (h @ w[n + "_proj.weight"].double().T for n in "qkv")
    q = _rms(q.unflatten(1, (H, D)), w["q_norm.weight"].double())
    k = _rms(k.unflatten(1, (G, D)), w["k_norm.weight"].double())
    v = v.unflatten(1, (G, D))
    for (c, n), old in zip(spans, cached):
        qi, ki, vi = _turn(q[at:at + n], c, 1e6, False), _turn(k[at:at + n], c, 1e6, False), v[at:at + n]
        if c:
            ki, vi = torch.cat([old[0].double(), ki]), torch.cat([old[1].double(), vi])
        o = torch.empty((n, H, D), device=DEV, dtype=torch.float64)
        for x in range(H):
            g = x // (H // G)
            o[:, x] = _softmax_sum(qi[:, x], ki[:, g], vi[:, g], c, D ** -0.5)
        out.append(o.flatten(1))
        at += n
    return torch.cat(out) @ w["o_proj.weight"].double().T


def _exact_mlp(h, w):
    g, u = h @ w["gate_proj.weight"].double().T, h @ w["up_proj.weight"].double().T
    return (torch.nn.functional.silu(g) * u) @ w["down_proj.weight"].double().T


def _exact_step(case, seed):
    W, H, G, _F, tied = DENSE[case["size"]]
    w = _weights(case, seed)
    ids, cached = _inputs(case, seed)
    new = _numbers(case["new"])
    spans = list(zip(_numbers(case["context"]), new))
    x = w["model.embed_tokens.weight"][torch.tensor(ids, device=DEV)].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        own = {n[len(p):]: t for n, t in w.items() if n.startswith(p)}
        att = {n[len("self_attn."):]: t for n, t in own.items() if n.startswith("self_attn.")}
        mlp = {n[len("mlp."):]: t for n, t in own.items() if n.startswith("mlp.")}
        x = x + _exact_attention(_rms(x, own["input_layernorm.weight"].double()), att, H, G, spans,
                                 [c if c is None else c[i] for c in cached])
        x = x + _exact_mlp(_rms(x, own["post_attention_layernorm.weight"].double()), mlp)
    last = torch.tensor(new, device=DEV).cumsum(0) - 1
    x = _rms(x[last], w["model.norm.weight"].double())
    head = w["model.embed_tokens.weight" if tied else "lm_head.weight"]
    return torch.cat([x @ part.double().T for part in head.split(16384)], dim=1)


def _exact_latent(case, h, w):
    z = LATENT[case["size"]]
    H, D, R, scale = z["heads"], 128, 512, 192 ** -0.5
    c_q = _rms(h @ w["dq"].double().T, w["dq.norm"].double())
    q = (c_q @ w["uq"].double().T).unflatten(1, (H, D + 64))
    down = h @ w["dkv"].double().T
    c = _rms(down[:, :R], w["dkv.norm"].double())
    k = (c @ w["uk"].double().T).unflatten(1, (H, D))
    v = (c @ w["uv"].double().T).unflatten(1, (H, D))
    out, at = torch.empty((h.shape[0], H, D), device=DEV, dtype=torch.float64), 0
    for n in _numbers(case["new"]):
        r = slice(at, at + n)
        k_rot = _turn(down[r, None, R:], 0, 1e4, True)[:, 0]
        q_rot = _turn(q[r, :, D:], 0, 1e4, True)
        for x in range(H):
            out[r, x] = _softmax_sum(torch.cat([q[r, x, :D], q_rot[:, x]], 1), torch.cat([k[r, x], k_rot], 1), v[r, x], 0, scale,
                                     window=z["window"], sink=w["sink"][x].double())
        at += n
    return dict(out=out.flatten(1) @ w["o"].double().T, pages=None)


def _exact_gla(case, h, w):
    H = GLA[case["size"]]["heads"]
    q, k = ((h @ w[n].double().T).unflatten(1, (H, 64)) for n in "qk")
    v = (h @ w["v"].double().T).unflatten(1, (H, 128))
    a = torch.sigmoid((h @ w["a1"].double().T) @ w["a2"].double().T + w["a2.b"].double()).pow(1.0 / 16.0).unflatten(1, (H, 64))
    outs, states, at = [], [], 0
    for n in _numbers(case["new"]):
        s = torch.zeros((H, 64, 128), device=DEV, dtype=torch.float64)
        for t in range(at, at + n):
            s = s * a[t, :, :, None] + k[t, :, :, None] * v[t, :, None, :]
            outs.append(torch.bmm(q[t, :, None, :] / 8.0, s)[:, 0])
        states.append(s)
        at += n
    o = _rms(torch.stack(outs), w["norm"].double()).flatten(1) * torch.nn.functional.silu(h @ w["g"].double().T)
    return dict(out=o @ w["o"].double().T, state=torch.stack(states))


def _exact_delta(case, h, w):
    z = DELTA[case["size"]]
    H, G, D = z["heads"], z["kv_heads"], 128
    x = h @ torch.cat([w["q"], w["k"], w["v"]]).double().T
    taps = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]).double()
    step = torch.nn.functional.softplus((h @ w["a1"].double().T) @ w["a2"].double().T + w["dt_bias"].double()).unflatten(1, (H, D))
    decay = torch.exp(-torch.exp(w["A_log"].double())[:, None] * step)
    beta = torch.sigmoid(h @ w["b"].double().T)
    gate = torch.sigmoid((h @ w["g1"].double().T) @ w["g2"].double().T)
    outs, states, at = [], [], 0
    for n in _numbers(case["new"]):
        past = torch.nn.functional.pad(x[at:at + n], (0, 0, 3, 0))
        y = torch.nn.functional.silu(sum(past[i:i + n] * taps[:, i] for i in range(4)))
        q, k, v = y.split([G * D, G * D, H * D], dim=1)
        q, k = (t.unflatten(1, (G, D)) for t in (q, k))
        q, k = (t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = ((t * f).repeat_interleave(H // G, dim=1) for t, f in ((q, D ** -0.5), (k, 1.0)))
        v = v.unflatten(1, (H, D))
        s = torch.zeros((H, D, D), device=DEV, dtype=torch.float64)
        for t in range(n):
            s = s * decay[at + t, :, :, None]
            u = beta[at + t][:, None] * (v[t] - torch.bmm(k[t, :, None, :], s)[:, 0])
            s = s + k[t, :, :, None] * u[:, None, :]
            outs.append(torch.bmm(q[t, :, None, :], s)[:, 0])
        states.append(s)
        at += n
    o = _rms(torch.stack(outs), w["norm"].double()).flatten(1) * gate
    return dict(out=o @ w["o"].double().T, state=torch.stack(states), ring=None)


def _exact_diff(case, h, w):
    z = DIFF[case["size"]]
    H, G = z["heads"], z["kv_heads"]
    q = _rms((h @ w["q"].double().T).unflatten(1, (H, 2, 64)), w["q.norm"].double())
    k = _rms((h @ w["k"].double().T).unflatten(1, (G, 2, 64)), w["k.norm"].double())
    v = (h @ w["v"].double().T).unflatten(1, (G, 128))
    lam = torch.exp((w["lq1"].double() * w["lk1"].double()).sum()) - torch.exp((w["lq2"].double() * w["lk2"].double()).sum()) + 0.6
    out, at = torch.empty((h.shape[0], H, 128), device=DEV, dtype=torch.float64), 0
    for n in _numbers(case["new"]):
        r = slice(at, at + n)
        for x in range(H):
            g = x // (H // G)
            a = [_softmax_sum(q[r, x, m], k[r, g, m], v[r, g], 0, 64 ** -0.5, chunk=2048) for m in (0, 1)]
            out[r, x] = _rms(a[0] - lam * a[1]) * 0.4
        at += n
    return dict(out=out.flatten(1) @ w["o"].double().T, keys=None, values=None)


def _exact_experts(case, h, w):
    z = EXPERTS[case["size"]]
    score = h @ w["router"].double().T
    top, chosen = score.topk(z["top"], dim=1)
    clamped = case["unit"] == "clamped"
    weight = torch.sigmoid(top) if clamped else torch.softmax(top, dim=1)

    def unit(x, name):
        u = x @ w[name + ".up"].double().T
        if not clamped:
            return torch.relu(u).square() @ w[name + ".down"].double().T
        g = (x @ w[name + ".gate"].double().T).clamp(max=7.0)
        return (g * torch.sigmoid(1.702 * g) * (u.clamp(-7.0, 7.0) + 1.0)) @ w[name + ".down"].double().T

    out = unit(h, "shared")
    if not clamped:
        out = out * torch.sigmoid(h @ w["shared.sg"].double().T)
    for e in range(z["experts"]):
        rows, place = torch.nonzero(chosen == e, as_tuple=True)
        f = weight[rows, place][:, None]
        y = unit(h[rows] * f, f"e{e}") if clamped else f * unit(h[rows], f"e{e}")
        out = out.index_add(0, rows, y)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    w = _weights(case, seed)
    h, cached = _inputs(case, seed)
    h = h.double()
    if kind == "mlp":
        return _exact_mlp(h, w)
    if kind == "attention":
        _W, H, G, _F, _ = DENSE[case["size"]]
        spans = list(zip(_numbers(case["context"]), _numbers(case["new"])))
        return dict(out=_exact_attention(h, w, H, G, spans, [c if c is None else c[0] for c in cached]), keys=None, values=None)
    return {"latent": _exact_latent, "gla": _exact_gla, "delta": _exact_delta, "diff": _exact_diff, "experts": _exact_experts}[kind](case, h, w)
