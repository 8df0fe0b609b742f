"""The work this framework is measured by: single layers through the parts' own entry points, and whole steps through
`Engine.step`, at the layer sizes `bench.py` knows, with random weights and inputs.

A case is a dict: `kind` (below), `size` (a row of SIZES) and the shape of the step.  All requests of a step are a
little ragged, as a continuous batch is.

=================  =============================================================================================
kind               what runs
=================  =============================================================================================
``model``          every layer of the Qwen2 decoder: packing, kernels, 32-bit logits (steps replayed from graphs)
``attention``      `GQAttention`: projections, rotation, paged cache write, attention, output projection
``mlp``            `GatedMLP`
``experts``        `RoutedExperts`: router, grouped products, weighted sum, gated shared expert
``general_delta``  the generalized delta rule with its projections (`GeneralDelta`)
``gated_delta``    the gated delta rule with its projections and convolutions (`GatedDelta`)
``selective``      the selective scan with its projections and convolution (`SelectiveScanMixer`)
``memory``         the matrix memory with exponential gates (`MatrixMemory`)
=================  =============================================================================================
"""
from __future__ import annotations

import math

import numpy as np
import torch

# Layer sizes: width, feed-forward, attention heads, mixers' heads and sizes, experts (bench.py's shapes of these names).
SIZES = {
    "0.5B": dict(hidden=896, ff=4864, vocab=151936, heads=14, kv_heads=2, dim=64, layers=24, expert_ff=1536, shared_ff=1792,
                 inner=1792, dt_rank=56, delta_heads=14, delta_kv=7, delta_dim=64, decay_rank=64),
    "1.5B": dict(hidden=1536, ff=8960, vocab=151936, heads=12, kv_heads=2, dim=128, layers=28, expert_ff=2816, shared_ff=3328,
                 inner=3072, dt_rank=96, delta_heads=12, delta_kv=6, delta_dim=128, decay_rank=96),
    "7B": dict(hidden=3584, ff=18944, vocab=152064, heads=28, kv_heads=4, dim=128, layers=28),
}
EXPERTS, TOP, STATE, TAPS, PAGE = 8, 2, 16, 4, 16
THETA, EPS, GATE_CAP, FLOOR, DECAY_RATE, UNIT_EPS = 1e6, 1e-6, 15.0, 1e-6, math.exp(-0.5), 1e-6
RECURRENT = ("general_delta", "gated_delta", "selective", "memory")


def listed():
    return [
        # serving: a decode step of a few conversations of the headline model, replayed from its graph
        dict(name="decode step, batch 8", kind="model", size="0.5B", requests=8, tokens=1, past=520),
        # serving: the headline model reads a long prompt
        dict(name="prompt step, 2048", kind="model", size="0.5B", requests=1, tokens=2048, past=0),
        # serving a large model: a full batch decodes over long contexts
        dict(name="attention, decode 32 x 4096", kind="attention", size="7B", dtype="bf16", portions=0, tokens=1, singles=32, past=4096),
        # continuous batching: portions of two prompts beside requests that decode
        dict(name="attention, mixed step", kind="attention", size="1.5B", dtype="bf16", portions=2, tokens=411, singles=5, past=700),
        # the true 32-bit path: one prompt
        dict(name="attention, 32-bit prompt", kind="attention", size="0.5B", dtype="f32", portions=1, tokens=517, singles=0, past=0),
        # a portion of a chunked prompt through a dense feed-forward
        dict(name="mlp, 300 tokens", kind="mlp", size="1.5B", dtype="bf16", tokens=300),
        # the true 32-bit path: its feed-forward
        dict(name="mlp, 32-bit", kind="mlp", size="0.5B", dtype="f32", tokens=517),
        # a prompt through routed experts
        dict(name="experts, 1500 tokens", kind="experts", size="0.5B", tokens=1500),
        # prompts through the recurrent mixers: one long prompt, or a batch of short ones; first or later portions
        dict(name="general delta, 3 prompts", kind="general_delta", size="0.5B", requests=3, tokens=500, past=0),
        dict(name="gated delta, 2048", kind="gated_delta", size="0.5B", requests=1, tokens=2048, past=0),
        dict(name="selective scan, 2048", kind="selective", size="0.5B", requests=1, tokens=2048, past=512),
        dict(name="matrix memory, 2 prompts", kind="memory", size="0.5B", requests=2, tokens=1000, past=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("model", "attention", "attention", "attention", "mlp", "mlp", "experts") + RECURRENT)
    if kind == "model":
        if rng.random() < 0.5:
            return dict(kind=kind, size="0.5B", requests=_log(rng, 1, 48), tokens=1, past=_log(rng, 40, 1000))
        requests = rng.randint(1, 3)
        return dict(kind=kind, size="0.5B", requests=requests, tokens=_log(rng, 60, 2000 // requests), past=rng.choice((0, _log(rng, 30, 900))))
    if kind == "attention":
        dtype = rng.choice(("bf16", "bf16", "f32"))
        if dtype == "f32":
            return dict(kind=kind, size="0.5B", dtype=dtype, portions=rng.randint(1, 2), tokens=_log(rng, 20, 350), singles=rng.randint(0, 4), past=_log(rng, 1, 300))
        if rng.random() < 0.4:
            size = rng.choice(("0.5B", "1.5B", "7B"))
            return dict(kind=kind, size=size, dtype=dtype, portions=0, tokens=1, singles=_log(rng, 2, 32), past=_log(rng, 60, 4000))
        size = rng.choice(("0.5B", "1.5B"))
        return dict(kind=kind, size=size, dtype=dtype, portions=rng.randint(1, 3), tokens=_log(rng, 65, 680), singles=rng.randint(0, 8), past=_log(rng, 1, 1000))
    if kind == "mlp":
        dtype = rng.choice(("bf16", "f32"))
        size = "0.5B" if dtype == "f32" else rng.choice(("0.5B", "1.5B", "7B"))
        return dict(kind=kind, size=size, dtype=dtype, tokens=_log(rng, 8, 517 if dtype == "f32" else 1024))
    size = rng.choice(("0.5B", "0.5B", "1.5B"))
    if kind == "experts":
        return dict(kind=kind, size=size, tokens=_log(rng, 24, 1500))
    requests = _log(rng, 1, 8)
    return dict(kind=kind, size=size, requests=requests, tokens=_log(rng, 100, 2048 // requests), past=rng.choice((0, _log(rng, 16, 1000))))


# ----------------------------------------------------------------------------------------
# The step's shape and its random numbers, the same for the framework and for the 64-bit restatement
# ----------------------------------------------------------------------------------------
def shape_of(case):
    """(new tokens per request, positions held before per request)"""
    if case["kind"] in ("mlp", "experts"):
        return [case["tokens"]], [0]
    if case["kind"] == "attention":
        p, s, past = case["portions"], case["singles"], case["past"]
        return ([max(2, case["tokens"] - 5 * i) for i in range(p)] + [1] * s,
                [max(0, past - 13 * i) for i in range(p)] + [max(1, past - 7 * i) for i in range(s)])
    n, past = case["requests"], case["past"]
    return [max(1, case["tokens"] - 3 * i) for i in range(n)], [max(0, past - 11 * i) for i in range(n)]


def torch_dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


class Numbers:
    """Random tensors of a seed, one after the other."""

    def __init__(self, seed, dtype):
        self.gen, self.dtype = torch.Generator(device="cuda").manual_seed(seed), dtype

    def normal(self, *shape, std=1.0, mean=0.0, dtype=None):
        t = torch.randn(shape, generator=self.gen, device="cuda", dtype=torch.float32)
        return t.mul_(std).add_(mean).to(dtype or self.dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, generator=self.gen, device="cuda", dtype=torch.float32).mul_(hi - lo).add_(lo)

    def matrix(self, rows, cols, gain=1.0):
        return self.normal(rows, cols, std=gain / math.sqrt(cols))

    def gain(self, n):
        return self.normal(n, std=0.1, mean=1.0)

    def step_bias(self, n):
        """The inverse softplus of step sizes spread evenly over the logarithm from 1e-3 to 1e-1."""
        dt = torch.exp(self.uniform(math.log(1e-3), math.log(1e-1), n))
        return (dt + torch.log(-torch.expm1(-dt))).to(self.dtype)


def attention_weights(num, z, prefix="", gain=1.0):
    h, nq, nkv, d = z["hidden"], z["heads"], z["kv_heads"], z["dim"]
    w = {"q_proj.weight": num.matrix(nq * d, h, 1.4), "k_proj.weight": num.matrix(nkv * d, h, 1.4),
         "v_proj.weight": num.matrix(nkv * d, h), "o_proj.weight": num.matrix(h, nq * d, gain),
         "q_proj.bias": num.normal(nq * d, std=0.3), "k_proj.bias": num.normal(nkv * d, std=0.3),
         "v_proj.bias": num.normal(nkv * d, std=0.1)}
    return {prefix + k: v for k, v in w.items()}


def mlp_weights(num, z, prefix="", gain=1.0):
    h, f = z["hidden"], z["ff"]
    return {prefix + "gate_proj.weight": num.matrix(f, h), prefix + "up_proj.weight": num.matrix(f, h),
            prefix + "down_proj.weight": num.matrix(h, f, gain)}


def layer_inputs(case, seed):
    """(weights by tensor name, rows of the step, what earlier portions of the requests left)"""
    z, num, kind = SIZES[case["size"]], Numbers(seed, torch_dtype(case)), case["kind"]
    q_lens, past = shape_of(case)
    h, requests, held = z["hidden"], len(q_lens), {}
    x = num.normal(sum(q_lens), h)
    if kind == "attention":
        w = attention_weights(num, z)
        held = {"k": num.normal(sum(past), z["kv_heads"], z["dim"], std=1.4), "v": num.normal(sum(past), z["kv_heads"], z["dim"])}
    elif kind == "mlp":
        w = mlp_weights(num, z)
    elif kind == "experts":
        f, s = z["expert_ff"], z["shared_ff"]
        w = {"router": num.matrix(EXPERTS, h), "shared.sg": num.matrix(1, h), "shared.gate": num.matrix(s, h),
             "shared.up": num.matrix(s, h), "shared.down": num.matrix(h, s)}
        for e in range(EXPERTS):
            w.update({f"e{e}.gate": num.matrix(f, h), f"e{e}.up": num.matrix(f, h), f"e{e}.down": num.matrix(h, f)})
    elif kind == "general_delta":
        H, D, R = z["delta_heads"], z["delta_dim"], z["decay_rank"]
        w = {n: num.matrix(H * D, h) for n in ("r", "k", "v", "g", "a")}
        w.update({"a.b": num.normal(H * D, std=0.5), "w1": num.matrix(R, h), "w2": num.matrix(H * D, R),
                  "w0": num.normal(H * D, mean=-3.0), "norm": num.gain(H * D), "o": num.matrix(h, H * D)})
        held = {"state": [(H, D, D)]}
    elif kind == "gated_delta":
        H, G, D = z["delta_heads"], z["delta_kv"], z["delta_dim"]
        w = {}
        for n, rows in (("q", G * D), ("k", G * D), ("v", H * D)):
            w[n], w[n + ".conv"] = num.matrix(rows, h), num.normal(rows, TAPS, std=0.5)
        w.update({"g": num.matrix(H * D, h), "b": num.matrix(H, h), "a": num.matrix(H, h),
                  "A_log": torch.log(num.uniform(1.0, 16.0, H)).to(num.dtype), "dt_bias": num.step_bias(H), "norm": num.gain(D),
                  "o": num.matrix(h, H * D)})
        held = {"state": [(H, D, D), (TAPS - 1, (2 * G + H) * D)]}
    elif kind == "selective":
        inner, R = z["inner"], z["dt_rank"]
        w = {"in": num.matrix(2 * inner, h), "conv": num.normal(inner, TAPS, std=0.5), "conv.b": num.normal(inner, std=0.1),
             "x": num.matrix(R + 2 * STATE, inner), "dt": num.matrix(inner, R, 0.5), "dt.b": num.step_bias(inner),
             "A_log": torch.log(torch.arange(1, STATE + 1, device="cuda", dtype=torch.float32)).repeat(inner, 1).to(num.dtype),
             "D": num.gain(inner), "o": num.matrix(h, inner)}
        held = {"state": [(inner, STATE), (TAPS - 1, inner)]}
    else:
        H, D = z["delta_heads"], z["delta_dim"]
        w = {"q": num.matrix(H * D, h), "k": num.matrix(H * D, h), "v": num.matrix(H * D, h), "g": num.matrix(H * D, h),
             "o": num.matrix(h, H * D), "norm": num.gain(H * D), "i": num.matrix(H, h, 0.5), "i.b": num.normal(H, std=0.1, mean=-1.0),
             "f": num.matrix(H, h, 0.5), "f.b": (3.0 + 3.0 * torch.arange(H, device="cuda") / max(1, H - 1)).to(num.dtype)}
        held = {"state": [(H, D, (D + 4) // 4 * 4), (H,)]}
    if "state" in held:      # zeros for a new request, else what a portion before this one may have left
        states = [num.normal(requests, *s, std=0.5, dtype=torch.float32) * (case["past"] > 0) for s in held["state"]]
        if kind == "memory":
            states[0][..., z["delta_dim"] + 1:] = 0.0       # padding of the value rows
        held = {"state": states}
    return w, x, held


def model_config(case):
    z = SIZES[case["size"]]
    return dict(architectures=["Qwen2ForCausalLM"], model_type="qwen2", vocab_size=z["vocab"], hidden_size=z["hidden"],
                intermediate_size=z["ff"], num_hidden_layers=z["layers"], num_attention_heads=z["heads"],
                num_key_value_heads=z["kv_heads"], rms_norm_eps=EPS, rope_theta=THETA, max_position_embeddings=4096,
                hidden_act="silu", tie_word_embeddings=True, use_sliding_window=False, eos_token_id=151645)


def model_inputs(case, seed):
    """(weights by tensor name, token ids per request, keys and values held before, per layer)"""
    z, num = SIZES[case["size"]], Numbers(seed, torch.bfloat16)
    q_lens, past = shape_of(case)
    w = {"model.embed_tokens.weight": num.normal(z["vocab"], z["hidden"]), "model.norm.weight": num.gain(z["hidden"])}
    held = []
    for i in range(z["layers"]):
        p = f"model.layers.{i}."
        # the last products are drawn smaller the deeper the model, so that the stream grows as in a trained one
        w.update(attention_weights(num, z, p + "self_attn.", gain=(2 * z["layers"]) ** -0.5))
        w.update(mlp_weights(num, z, p + "mlp.", gain=(2 * z["layers"]) ** -0.5))
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = num.gain(z["hidden"]), num.gain(z["hidden"])
        held.append((num.normal(sum(past), z["kv_heads"], z["dim"], std=1.4), num.normal(sum(past), z["kv_heads"], z["dim"])))
    rng = np.random.default_rng(seed)
    ids = [[int(t) for t in rng.integers(0, z["vocab"], n)] for n in q_lens]
    return w, ids, held


def pages_of(case):
    """(block table [requests, width] int32 with pages in no particular order, number of pages)"""
    q_lens, past = shape_of(case)
    blocks = [-(-(n + p) // PAGE) for n, p in zip(q_lens, past)]
    order = np.random.default_rng(sum(blocks)).permutation(sum(blocks))
    table = -np.ones((len(blocks), (max(blocks) + 7) & ~7), dtype=np.int32)
    at = 0
    for r, b in enumerate(blocks):
        table[r, :b] = order[at: at + b]
        at += b
    return table, sum(blocks)


def rows_of(lens, first):
    """(request of each row, position of each row)"""
    return (np.concatenate([np.full(n, r, dtype=np.int64) for r, n in enumerate(lens)]),
            np.concatenate([np.arange(p, p + n) for n, p in zip(lens, first)]))


def put_pages(cache, table, lens, first, rows):
    """rows [tokens, kv heads, dim] of positions first.. of each request into their pages."""
    req, pos = rows_of(lens, first)
    page = torch.from_numpy(table[req, pos // PAGE].astype(np.int64)).cuda()
    cache[page, :, torch.from_numpy(pos % PAGE).cuda()] = rows.to(cache.dtype)


# ----------------------------------------------------------------------------------------
# The framework
# ----------------------------------------------------------------------------------------
def part_spec(case):
    from llm_inference_lab_b200.parts.spec import PartSpec

    z, kind = SIZES[case["size"]], case["kind"]
    if kind == "attention":
        rope = PartSpec("rope", {"theta": THETA, "rotary_dim": z["dim"]})
        return "mixer", PartSpec("gqa_attention", dict(hidden=z["hidden"], n_heads=z["heads"], n_kv_heads=z["kv_heads"], head_dim=z["dim"],
                                                       qkv_bias=True, out_bias=False, window=0, position=rope))
    if kind == "mlp":
        return "feed_forward", PartSpec("gated_mlp", dict(hidden=z["hidden"], intermediate=z["ff"], act="silu"))
    if kind == "experts":
        return "feed_forward", PartSpec("routed_experts", dict(hidden=z["hidden"], experts=EXPERTS, top=TOP, expert_ff=z["expert_ff"],
                                                               shared_ff=z["shared_ff"], shared_gate=True))
    if kind == "general_delta":
        return "mixer", PartSpec("general_delta", dict(hidden=z["hidden"], heads=z["delta_heads"], dim=z["delta_dim"], eps=EPS,
                                                       decay_rate=DECAY_RATE, decay_rank=z["decay_rank"]))
    if kind == "gated_delta":
        return "mixer", PartSpec("gated_delta", dict(hidden=z["hidden"], heads=z["delta_heads"], kv_heads=z["delta_kv"], dim=z["delta_dim"],
                                                     vdim=z["delta_dim"], taps=TAPS, eps=EPS, unit_eps=UNIT_EPS))
    if kind == "selective":
        return "mixer", PartSpec("selective_scan", dict(hidden=z["hidden"], inner=z["inner"], state=STATE, dt_rank=z["dt_rank"], taps=TAPS))
    return "mixer", PartSpec("matrix_memory", dict(hidden=z["hidden"], heads=z["delta_heads"], dim=z["delta_dim"], vdim=z["delta_dim"],
                                                   gate_cap=GATE_CAP, eps=EPS, floor=FLOOR))


def step_context(case, dtype):
    from llm_inference_lab_b200.parts.base import GroupView, StepContext

    q_lens, past = shape_of(case)
    kv = [n + p for n, p in zip(q_lens, past)]
    table, _ = pages_of(case)
    req, pos = rows_of(q_lens, past)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()  # noqa: E731
    group = GroupView(PAGE, 0, t(table[req, pos // PAGE] * PAGE + pos % PAGE), t(table))
    return StepContext(dtype=dtype, device=torch.device("cuda:0"), n_tokens=sum(q_lens), n_requests=len(q_lens),
                       token_ids=t(np.zeros(sum(q_lens))), row_req=t(req), row_pos=t(pos),
                       q_start=t(np.concatenate([[0], np.cumsum(q_lens)])), kv_len=t(kv), pos0=t(past),
                       state_slot=t(np.arange(len(q_lens))), groups=[group], q_lens=q_lens, kv_lens=kv,
                       state_slots=list(range(len(q_lens))), max_q_len=max(q_lens), max_kv_len=max(kv))


def prepare(case, seed):
    if case["kind"] == "model":
        return prepare_model(case, seed)
    import llm_inference_lab_b200.models.builder  # noqa: F401  (registers the parts)
    from llm_inference_lab_b200.parts.base import CacheView, lookup
    from llm_inference_lab_b200.parts.spec import CacheParts

    dtype, z = torch_dtype(case), SIZES[case["size"]]
    w, x, held = layer_inputs(case, seed)
    family, spec = part_spec(case)
    part = lookup(family, spec.kind)(spec, w, dtype, torch.device("cuda:0"))
    ctx = step_context(case, dtype)
    cache, outs = None, []
    if case["kind"] == "attention":
        table, pages = pages_of(case)
        k, v = (torch.zeros((pages, z["kv_heads"], PAGE, z["dim"]), dtype=dtype, device="cuda") for _ in range(2))
        _, past = shape_of(case)
        put_pages(k, table, past, [0] * len(past), held["k"])
        put_pages(v, table, past, [0] * len(past), held["v"])
        cache, outs = CacheView(part.cache_need(spec), group=0, k=k, v=v), [k, v]
    elif "state" in held:
        need, outs = part.cache_need(spec), held["state"]
        if isinstance(need, CacheParts):
            cache = CacheView(need, parts=[CacheView(n, state=s) for n, s in zip(need.parts, outs)])
        else:
            cache = CacheView(need, state=outs[0])
    return {"case": case, "part": part, "x": x, "ctx": ctx, "cache": cache, "outs": outs}


def prepare_model(case, seed):
    from llm_inference_lab_b200.engine import Engine, Entry
    from llm_inference_lab_b200.models.builder import CausalLM
    from llm_inference_lab_b200.registry import resolve

    w, ids, held = model_inputs(case, seed)
    q_lens, past = shape_of(case)
    cfg = model_config(case)
    arch = resolve(cfg)
    model = CausalLM(arch.blueprint(arch.config_class.from_dict(cfg)), w, torch.bfloat16, torch.device("cuda:0"))
    pages = sum(-(-(n + p) // PAGE) + 1 for n, p in zip(q_lens, past))
    engine = Engine(model, "bf16", max_tokens=pages * PAGE, page_size=PAGE, max_requests=max(8, len(q_lens)),
                    max_batch_tokens=max(512, sum(q_lens)))
    engine.enable_step_graphs()
    for r, p in enumerate(past):
        engine.open(r)
        if p:
            engine.cache.reserve(r, p)
            engine.cache.commit(r, p)
    table = -np.ones((len(past), max(1, -(-max(past) // PAGE))), dtype=np.int32)
    for r in range(len(past)):
        row = engine.cache.block_table(r, 0)[: table.shape[1]]
        table[r, : len(row)] = row
    for view, (k, v) in zip(engine.views, held):
        view.k.zero_(), view.v.zero_()
        put_pages(view.k, table, past, [0] * len(past), k)
        put_pages(view.v, table, past, [0] * len(past), v)
    entries = [Entry(r, t, [len(t) - 1]) for r, t in enumerate(ids)]
    outs = [t for view in engine.views for t in (view.k, view.v)]
    return {"case": case, "engine": engine, "entries": entries, "lens": q_lens, "outs": outs}


def run(state):
    if "engine" in state:
        engine = state["engine"]
        for r, n in enumerate(state["lens"]):
            engine.cache.reserve(r, n)
        logits = engine.step(state["entries"], reserved=True)
        for r in range(len(state["lens"])):
            engine.cache.rollback(r)      # the next pass is this step once more
        return [logits] + state["outs"]
    part, x, ctx = state["part"], state["x"], state["ctx"]
    ctx.scratch.clear()                   # a step's own buffers
    y = part.forward(x, ctx) if state["cache"] is None else part.forward(x, ctx, state["cache"])
    if y.dim() == 3:                      # a product may come as partial sums, which its consumer adds
        y = y.sum(0)
    return [y] + state["outs"]


# ----------------------------------------------------------------------------------------
# What a pass cannot do without
# ----------------------------------------------------------------------------------------
def attention_work(z, q_lens, past, b):
    h, nq, nkv, d, T = z["hidden"], z["heads"], z["kv_heads"], z["dim"], sum(q_lens)
    keys = sum(n + p for n, p in zip(q_lens, past))
    seen = sum(n * p + n * (n + 1) / 2 for n, p in zip(q_lens, past))
    weights = h * (2 * nq + 2 * nkv) * d
    return b * (weights + 2 * T * h + 2 * nkv * d * (keys + T)), 2 * T * weights + 4 * seen * nq * d


def work(case):
    z, kind = SIZES[case["size"]], case["kind"]
    b = 4 if case.get("dtype") == "f32" else 2
    q_lens, past = shape_of(case)
    h, T, R = z["hidden"], sum(q_lens), len(q_lens)
    if kind == "model":
        nb, nf = attention_work(z, q_lens, past, b)
        nb += b * 3 * h * z["ff"] - b * 2 * T * h
        nf += 6 * T * h * z["ff"]
        return {"bytes": z["layers"] * nb + b * z["vocab"] * h + 4 * R * z["vocab"], "flops": z["layers"] * nf + 2 * R * h * z["vocab"]}
    if kind == "attention":
        nb, nf = attention_work(z, q_lens, past, b)
        return {"bytes": nb, "flops": nf}
    if kind == "mlp":
        return {"bytes": b * (3 * h * z["ff"] + 2 * T * h), "flops": 6 * T * h * z["ff"]}
    if kind == "experts":
        f, s = z["expert_ff"], z["shared_ff"]
        return {"bytes": 2 * h * (EXPERTS + 1 + 3 * EXPERTS * f + 3 * s) + 6 * T * h,
                "flops": 2 * T * h * (EXPERTS + 1) + 6 * T * h * (TOP * f + s)}
    if kind == "selective":
        inner, rank = z["inner"], z["dt_rank"]
        weights = 3 * h * inner + inner * (2 * rank + 2 * STATE)
        return {"bytes": 2 * weights + 6 * T * h + 8 * R * inner * (STATE + TAPS - 1), "flops": 2 * T * weights + 7 * T * inner * STATE}
    H, D = z["delta_heads"], z["delta_dim"]
    if kind == "general_delta":
        weights, per = h * (6 * H * D + z["decay_rank"]) + H * D * z["decay_rank"], 9
    elif kind == "gated_delta":
        weights, per = h * (3 * H * D + 2 * z["delta_kv"] * D + 2 * H), 7
    else:
        weights, per = h * (5 * H * D + 2 * H), 5
    return {"bytes": 2 * weights + 6 * T * h + 8 * R * H * D * D, "flops": 2 * T * weights + per * T * H * D * D}


def tolerance(case):
    """About four times what sums in another order gave (the plain kernels against the tensor cores; in 32-bit, the
    kernels against 64-bit): in 16-bit storage an intermediate result that is rounded the other way travels on, through
    all layers of a model, through the scores of an attention, or only through one projection."""
    kind = case["kind"]
    if kind == "model":
        return {"rel": 0.03, "max": 0.25}
    if case.get("dtype") == "f32":
        return {"rel": 8e-6, "max": 5e-5}
    return {"attention": {"rel": 0.014, "max": 0.08}, "mlp": {"rel": 7e-3, "max": 0.02},
            "experts": {"rel": 6e-4, "max": 0.016}}.get(kind, {"rel": 8e-4, "max": 0.03})


# ----------------------------------------------------------------------------------------
# The same in 64-bit, in plain torch
# ----------------------------------------------------------------------------------------
def rotate(x, pos):
    """Rotation of halves; frequencies and angles are 32-bit numbers, as the framework defines them."""
    d = x.shape[-1]
    freq = torch.from_numpy(np.power(THETA, -2.0 * np.arange(d // 2) / d).astype(np.float32)).cuda()
    angle = (torch.from_numpy(pos.astype(np.float32)).cuda()[:, None] * freq).double()[:, None, :]
    a, b = x[..., : d // 2], x[..., d // 2:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def exact_attention(w, x, z, q_lens, past, k_held, v_held, prefix=""):
    """(result, new keys, new values)"""
    g = lambda n: w[prefix + n].double()  # noqa: E731
    nq, nkv, d, T = z["heads"], z["kv_heads"], z["dim"], x.shape[0]
    _, pos = rows_of(q_lens, past)
    q = rotate((x @ g("q_proj.weight").T + g("q_proj.bias")).view(T, nq, d), pos)
    k = rotate((x @ g("k_proj.weight").T + g("k_proj.bias")).view(T, nkv, d), pos)
    v = (x @ g("v_proj.weight").T + g("v_proj.bias")).view(T, nkv, d)
    outs, at, held = [], 0, 0
    for n, p in zip(q_lens, past):
        kk, vv = torch.cat([k_held[held: held + p].double(), k[at: at + n]]), torch.cat([v_held[held: held + p].double(), v[at: at + n]])
        mask = torch.arange(n + p, device="cuda")[None, :] > torch.arange(p, p + n, device="cuda")[:, None]
        heads = []
        for h in range(nq):
            s = q[at: at + n, h] @ kk[:, h // (nq // nkv)].T / math.sqrt(d)
            heads.append(torch.softmax(s.masked_fill(mask, -math.inf), dim=-1) @ vv[:, h // (nq // nkv)])
        outs.append(torch.cat(heads, dim=-1))
        at, held = at + n, held + p
    return torch.cat(outs) @ g("o_proj.weight").T, k, v


def silu(x):
    return x * torch.sigmoid(x)


def gated(x, gate, up, down):
    return (silu(x @ gate.double().T) * (x @ up.double().T)) @ down.double().T


def norm(x, weight, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight.double()


def conv_silu(u, kept, taps, bias=None):
    """Causal convolution per channel over the last inputs, then SiLU; (result, the last taps - 1 inputs)."""
    full, n = torch.cat([kept.double(), u]), u.shape[0]
    out = sum(full[j: j + n] * taps[:, j].double() for j in range(TAPS))
    return silu(out if bias is None else out + bias.double()), full[-(TAPS - 1):]


def exact_model(case, seed):
    z = SIZES[case["size"]]
    w, ids, held = model_inputs(case, seed)
    q_lens, past = shape_of(case)
    x = w["model.embed_tokens.weight"][torch.tensor([t for row in ids for t in row], device="cuda")].double()
    for i, (k, v) in enumerate(held):
        p = f"model.layers.{i}."
        x = x + exact_attention(w, norm(x, w[p + "input_layernorm.weight"]), z, q_lens, past, k, v, p + "self_attn.")[0]
        x = x + gated(norm(x, w[p + "post_attention_layernorm.weight"]), *(w[p + f"mlp.{n}_proj.weight"] for n in ("gate", "up", "down")))
    last = torch.from_numpy(np.cumsum(q_lens) - 1).cuda()
    # (the pages' order is the cache manager's: the keys and values are not laid out here)
    return [norm(x[last], w["model.norm.weight"]) @ w["model.embed_tokens.weight"].double().T] + [None] * (2 * z["layers"])


def exact_recurrent(case, w, x, states):
    z, kind = SIZES[case["size"]], case["kind"]
    g = {n: t.double() for n, t in w.items()}
    H, D = z.get("delta_heads"), z.get("delta_dim")
    S, q_lens = [s.double().clone() for s in states], shape_of(case)[0]
    outs, at = [], 0
    for r, n in enumerate(q_lens):
        h = x[at: at + n]
        at += n
        state, rows = S[0][r], []
        if kind == "selective":
            inner, rank = z["inner"], z["dt_rank"]
            xz = h @ g["in"].T
            u, S[1][r] = conv_silu(xz[:, :inner], S[1][r], w["conv"], w["conv.b"])
            low = u @ g["x"].T
            dt = torch.nn.functional.softplus(low[:, :rank] @ g["dt"].T + g["dt.b"])
            B, C, A = low[:, rank: rank + STATE], low[:, rank + STATE:], -torch.exp(g["A_log"])
            for t in range(n):
                state = torch.exp(dt[t, :, None] * A) * state + (dt[t] * u[t])[:, None] * B[t]
                rows.append(state @ C[t])
            y = (torch.stack(rows) + g["D"] * u) * silu(xz[:, inner:])
        elif kind == "general_delta":
            q, k, v, gate, a = (h @ g[m].T for m in ("r", "k", "v", "g", "a"))
            decay = torch.exp(-DECAY_RATE * torch.sigmoid(torch.tanh(h @ g["w1"].T) @ g["w2"].T + g["w0"])).view(n, H, D)
            rate, (q, k, v) = torch.sigmoid(a + g["a.b"]).view(n, H, D), (m.view(n, H, D) for m in (q, k, v))
            unit = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
            for t in range(n):
                seen = (unit[t][:, :, None] * state).sum(1)
                state = decay[t][:, :, None] * state - (rate[t] * unit[t])[:, :, None] * seen[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
                rows.append((state * q[t][:, :, None]).sum(1))
            o = norm(torch.stack(rows), torch.ones(D, device="cuda")).reshape(n, H * D)
            y = o * g["norm"] * torch.sigmoid(gate)
        elif kind == "gated_delta":
            G = z["delta_kv"]
            u, S[1][r] = conv_silu(torch.cat([h @ g[m].T for m in ("q", "k", "v")], dim=1), S[1][r],
                                   torch.cat([w[m + ".conv"] for m in ("q", "k", "v")]))
            q, k, v = u[:, : G * D].view(n, G, D), u[:, G * D: 2 * G * D].view(n, G, D), u[:, 2 * G * D:].view(n, H, D)
            q, k = (m / torch.sqrt((m * m).sum(-1, keepdim=True) + UNIT_EPS) for m in (q, k))
            q, k = (m.repeat_interleave(H // G, dim=1) for m in (q * D ** -0.5, k))
            beta = torch.sigmoid(h @ g["b"].T)
            decay = torch.exp(-torch.exp(g["A_log"]) * torch.nn.functional.softplus(h @ g["a"].T + g["dt_bias"]))
            for t in range(n):
                state = decay[t][:, None, None] * state
                new = beta[t][:, None] * (v[t] - (state * k[t][:, :, None]).sum(1))
                state = state + k[t][:, :, None] * new[:, None, :]
                rows.append((state * q[t][:, :, None]).sum(1))
            y = norm(torch.stack(rows), w["norm"]).reshape(n, H * D) * silu(h @ g["g"].T)
        else:
            q, k, v, gate = (h @ g[m].T for m in ("q", "k", "v", "g"))
            q, k, v = (q * D ** -0.5).view(n, H, D), k.view(n, H, D), v.view(n, H, D)
            v = torch.cat([v, torch.ones(n, H, 1, device="cuda", dtype=torch.float64),
                           torch.zeros(n, H, state.shape[-1] - D - 1, device="cuda", dtype=torch.float64)], dim=-1)
            log_i = GATE_CAP * torch.tanh((h @ g["i"].T + g["i.b"]) / GATE_CAP)
            log_f = torch.nn.functional.logsigmoid(GATE_CAP * torch.tanh((h @ g["f"].T + g["f.b"]) / GATE_CAP))
            m = S[1][r]
            for t in range(n):
                top = torch.maximum(log_f[t] + m, log_i[t])
                state = torch.exp(log_f[t] + m - top)[:, None, None] * state + torch.exp(log_i[t] - top)[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
                m = top
                o = (state * q[t][:, :, None]).sum(1)
                rows.append(o[:, :D] / (torch.maximum(o[:, D].abs(), torch.exp(-m)) + FLOOR)[:, None])
            S[1][r] = m
            y = norm(torch.stack(rows), torch.ones(D, device="cuda")).reshape(n, H * D) * g["norm"] * torch.sigmoid(gate)
        S[0][r] = state
        outs.append(y @ g["o"].T)
    return [torch.cat(outs)] + S


def exact(case, seed):
    kind = case["kind"]
    if kind == "model":
        return exact_model(case, seed)
    z = SIZES[case["size"]]
    w, x, held = layer_inputs(case, seed)
    x = x.double()
    if kind == "mlp":
        return [gated(x, w["gate_proj.weight"], w["up_proj.weight"], w["down_proj.weight"])]
    if kind == "experts":
        scores = torch.softmax(x @ w["router"].double().T, dim=-1)
        best, chosen = scores.topk(TOP, dim=-1)
        best = best / best.sum(-1, keepdim=True)
        y = torch.sigmoid(x @ w["shared.sg"].double().T) * gated(x, w["shared.gate"], w["shared.up"], w["shared.down"])
        for e in range(EXPERTS):
            share = (best * (chosen == e)).sum(-1, keepdim=True)
            y = y + share * gated(x, w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"])
        return [y]
    if kind == "attention":
        q_lens, past = shape_of(case)
        table, pages = pages_of(case)
        y, k_new, v_new = exact_attention(w, x, z, q_lens, past, held["k"], held["v"])
        k, v = (torch.zeros((pages, z["kv_heads"], PAGE, z["dim"]), dtype=torch.float64, device="cuda") for _ in range(2))
        for cache, before, new in ((k, held["k"], k_new), (v, held["v"], v_new)):
            put_pages(cache, table, past, [0] * len(past), before)
            put_pages(cache, table, q_lens, past, new)
        return [y, k, v]
    return exact_recurrent(case, w, x, held["state"])
