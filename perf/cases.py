"""
The work this engine is asked to do, as cases that can be timed: whole decode steps of a Llama 3.2 1B sized model through
`StepRunner.step`, and the layers of the decoders it serves, each through its part's own `forward`: attention and
feed-forward of the Llama decoders in both activation dtypes, gated linear attention and retention, the gated delta rule,
attention over a cached latent, routed experts.  Weights and inputs are drawn from a seed on the GPU.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` builds what a program holds before the
call, `run` is one call, `exact` the same in 64 bits from plain torch, `work` what a call cannot do without.
"""

from __future__ import annotations

import math

import torch

from tinyserve_llm_b200.cache.manager import CacheManager, plan_layout
from tinyserve_llm_b200.cache.storage import DeviceCacheStorage, EntryBinding
from tinyserve_llm_b200.config.llama import LlamaConfig, llama_model_spec
from tinyserve_llm_b200.config.spec import (AttentionSpec, GatedDeltaRuleSpec, GatedMLPSpec, InlineRotarySpec, LatentAttentionSpec,
                                            LinearRecurrenceSpec, Llama3Scaling, RotarySpec, RoutedExpertsSpec)
from tinyserve_llm_b200.engine.step import HostView, StepContext, StepEntry, StepRunner
from tinyserve_llm_b200.ops import get_ops
from tinyserve_llm_b200.parts.base import Runtime, part_class
from tinyserve_llm_b200.parts.model import DecoderModel, declared_tensors

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
SCALING = {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
           "original_max_position_embeddings": 8192}
THETA = 500000.0
# Llama 3.2 1B, whose layer sizes the benchmark and most cases take; heads of 128 are those of Llama 3.2 3B and 3.1 8B
LLAMA_1B = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": 128256, "hidden_size": 2048,
            "intermediate_size": 8192, "num_hidden_layers": 16, "num_attention_heads": 32, "num_key_value_heads": 8,
            "head_dim": 64, "hidden_act": "silu", "rms_norm_eps": 1e-5, "rope_theta": THETA, "rope_scaling": SCALING,
            "max_position_embeddings": 16384, "tie_word_embeddings": True, "attention_bias": False, "mlp_bias": False}
PAGE = 256
NORM_EPS = 1e-6
DECAY_RANK, GATE_RANK, TAU, TAPS, UNIT_EPS = 16, 16, 16.0, 4, 1e-6
SWISH_LIMIT, SWISH_ALPHA = 7.0, 1.702


# ------------------------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # one user waiting for the next token: the smallest call of the engine, the benchmark's batch-1 point
        _step("decode_1x2048", 1, 2048),
        # the benchmark's headline: 8 requests that decode behind 4,096 tokens each
        _step("decode_8x4096", 8, 4096),
        # a whole prompt through a 1B model's attention layer (the benchmark's prefill length)
        _attention("attention_prompt_2048", "bf16", 2048, 32, 8, 64, 1, 2048, 0),
        # portions of odd lengths behind cached tokens in one step, heads of 128 (an 8B model's layer): chunked prefill and turns of a chat
        _attention("attention_portions_128", "bf16", 4096, 32, 8, 128, 3, 1531, 1000),
        # the 32-bit path of the whole model (correctness runs): a prompt of 512 tokens
        _attention("attention_f32_512", "f32", 2048, 32, 8, 64, 1, 512, 0),
        # feed-forward of a prompt, of a decode step of 64 requests, and of an odd-sized prompt in 32 bits
        _ffn("ffn_prompt_2048", "bf16", 2048, 8192, 2048),
        _ffn("ffn_64", "bf16", 2048, 8192, 64),
        _ffn("ffn_f32_100", "f32", 2048, 8192, 100),
        # gated linear attention over a whole prompt (Duduvik, medium size of the designs' comparison)
        _recurrence("gla_prompt_2048", "channel_logits", 2048, 8, 128, 256, 1, 2048),
        # the delta rule with a decay a channel over three prompt portions that carry their state on (Nipizen, medium)
        _delta("delta_portions", "channel", 2048, 8, 4, 128, 128, 3, 1001),
        # windowed attention over a cached latent, a whole prompt (Duduvik, medium)
        _latent("latent_prompt_2048", 2048, 16, 128, 64, 1536, 512, 1024, 1, 2048, 0),
        # routed experts and the shared one in a decode step of 8 requests (Duduvik, medium)
        _experts("experts_8", 2048, 32, 4, 1024, 2048, 8),
    ]


def draw(rng) -> dict:
    """One more case: kinds evenly, sizes over the logarithm of their range, odd ones among them."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("step", "attention", "ffn", "recurrence", "delta", "latent", "experts"))
    if kind == "step":
        requests = log(1, 64)
        return _step(None, requests, min(log(128, 8192), 32768 // requests))
    if kind == "attention":
        hidden, heads, kv_heads, dim = rng.choice(((2048, 32, 8, 64), (3072, 24, 8, 128), (4096, 32, 8, 128)))
        if rng.random() < 1 / 3:
            return _attention(None, "f32", 2048, 32, 8, 64, rng.randint(1, 4), log(1, 600), log(1, 400) if rng.random() < 0.5 else 0)
        requests = rng.randint(1, 6)
        return _attention(None, "bf16", hidden, heads, kv_heads, dim, requests, min(log(2, 2048), 4096 // requests),
                          log(1, 2048) if rng.random() < 0.5 else 0)
    if kind == "ffn":
        if rng.random() < 1 / 3:
            return _ffn(None, "f32", 2048, 8192, log(1, 300))
        hidden, ff = rng.choice(((2048, 8192), (3072, 8192), (4096, 14336)))
        return _ffn(None, "bf16", hidden, ff, min(log(1, 2048), 2048 * 2048 * 8192 // (hidden * ff)))
    if kind == "recurrence":
        heads = rng.choice((4, 8))
        requests = rng.randint(1, 4)
        return _recurrence(None, rng.choice(("channel_logits", "head")), 256 * heads, heads, 128, 256, requests, log(2, 2048 // requests))
    if kind == "delta":
        scope = rng.choice(("channel", "head"))
        requests = rng.randint(1, 4)
        heads = rng.choice((4, 8)) if scope == "channel" else rng.choice((8, 16))
        return _delta(None, scope, (256 if scope == "channel" else 128) * heads, heads, max(1, heads // (2 if scope == "channel" else 4)),
                      128, 128, requests, log(2, 2048 // requests))
    if kind == "latent":
        heads = rng.choice((8, 16))
        requests = rng.randint(1, 3)
        return _latent(None, 128 * heads, heads, 128, 64, 96 * heads, 512, rng.choice((0, 1024)), requests, log(2, 2048 // requests),
                       log(1, 2048) if rng.random() < 0.5 else 0)
    experts, hidden = rng.choice(((16, 1024), (32, 2048)))
    return _experts(None, hidden, experts, 4, hidden // 2, hidden, log(1, 2048))


def _case(name, **values) -> dict:
    return dict({"name": name} if name else {}, **values)


def _step(name, requests, context):
    return _case(name, kind="step", requests=requests, context=context)


def _attention(name, dtype, hidden, heads, kv_heads, dim, requests, tokens, cached):
    return _case(name, kind="attention", dtype=dtype, hidden=hidden, heads=heads, kv_heads=kv_heads, dim=dim, requests=requests,
                 tokens=tokens, cached=cached)


def _ffn(name, dtype, hidden, ff, rows):
    return _case(name, kind="ffn", dtype=dtype, hidden=hidden, ff=ff, rows=rows)


def _recurrence(name, decay, hidden, heads, dim, vdim, requests, tokens):
    return _case(name, kind="recurrence", decay=decay, hidden=hidden, heads=heads, dim=dim, vdim=vdim, requests=requests, tokens=tokens)


def _delta(name, scope, hidden, heads, kv_heads, dim, vdim, requests, tokens):
    return _case(name, kind="delta", scope=scope, hidden=hidden, heads=heads, kv_heads=kv_heads, dim=dim, vdim=vdim, requests=requests,
                 tokens=tokens)


def _latent(name, hidden, heads, dim, rot, q_rank, kv_rank, window, requests, tokens, cached):
    return _case(name, kind="latent", hidden=hidden, heads=heads, dim=dim, rot=rot, q_rank=q_rank, kv_rank=kv_rank, window=window,
                 requests=requests, tokens=tokens, cached=cached)


def _experts(name, hidden, experts, top, expert_ff, shared_ff, tokens):
    return _case(name, kind="experts", hidden=hidden, experts=experts, top=top, expert_ff=expert_ff, shared_ff=shared_ff, tokens=tokens)


def _lengths(case) -> tuple[list[int], list[int]]:
    """(tokens fed, tokens cached before) of each request: the first feeds `tokens`, each further one less."""
    n, tokens, cached = case["requests"], case["tokens"], case.get("cached", 0)
    return [max(1, tokens * (n - i) // n) for i in range(n)], [cached * (i + 1) // n for i in range(n)]


# ------------------------------------------------------------------------------------------------ inputs from the seed alone
def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, dtype, std=1.0) -> torch.Tensor:
    out = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(generator=g)
    return out.mul_(std).to(dtype)


def _uniform(g, shape, lo, hi) -> torch.Tensor:
    return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=g)


def _pages(g, contexts: list[int], page: int) -> tuple[torch.Tensor, int]:
    """Block tables over pages handed out in no particular order."""
    counts = [-(-n // page) for n in contexts]
    order = torch.randperm(sum(counts), generator=g, device=DEV).tolist()
    rows, width = [], max(counts)
    for n in counts:
        rows.append(order[:n] + [-1] * (width - n))
        order = order[n:]
    return torch.tensor(rows, dtype=torch.int32, device=DEV), sum(counts)


def _inputs(case, seed) -> dict:
    """Weights, activations, caches and states: plain tensors."""
    g, kind = _generator(seed), case["kind"]
    dtype = DTYPES[case.get("dtype", "bf16")]

    def w(*shape, std=0.02):
        return _normal(g, shape, dtype, std)

    if kind == "step":
        spec = llama_model_spec(LlamaConfig.from_dict(LLAMA_1B))
        weights = {name: (1 + _normal(g, d.shape, torch.float32, 0.01)).to(dtype) if d.init == "unit" else w(*d.shape)
                   for name, d in declared_tensors(spec).items()}
        tokens = torch.randint(0, spec.vocab_size, (case["requests"],), generator=g, device=DEV).tolist()
        pages = case["requests"] * (case["context"] // PAGE + 1)
        shape = (pages, 16, 8, PAGE, 64)
        return dict(spec=spec, weights=weights, tokens=tokens, pages=pages, keys=_normal(g, shape, dtype), values=_normal(g, shape, dtype))
    if kind == "ffn":
        H, I = case["hidden"], case["ff"]
        return dict(x=_normal(g, (case["rows"], H), dtype),
                    weights={"gate_proj.weight": w(I, H), "up_proj.weight": w(I, H), "down_proj.weight": w(H, I)})
    if kind == "experts":
        H, E, F, S = case["hidden"], case["experts"], case["expert_ff"], case["shared_ff"]
        weights = {"router": w(E, H), "router.b": w(E)}
        for e in range(E):
            weights.update({f"e{e}.gate": w(F, H), f"e{e}.up": w(F, H), f"e{e}.down": w(H, F)})
        weights.update({"shared.gate": w(S, H), "shared.up": w(S, H), "shared.down": w(H, S)})
        return dict(x=_normal(g, (case["tokens"], H), dtype), weights=weights)
    fed, cached = _lengths(case)
    contexts = [a + b for a, b in zip(fed, cached)]
    out = dict(x=_normal(g, (sum(fed), case["hidden"]), dtype), fed=fed, cached=cached)
    H, D = case["heads"], case["dim"]
    if kind == "attention":
        out["weights"] = {"q_proj.weight": w(H * D, case["hidden"]), "k_proj.weight": w(case["kv_heads"] * D, case["hidden"]),
                          "v_proj.weight": w(case["kv_heads"] * D, case["hidden"]), "o_proj.weight": w(case["hidden"], H * D)}
        out["table"], pages = _pages(g, contexts, PAGE)
        shape = (pages, 1, case["kv_heads"], PAGE, D)
        out["keys"], out["values"] = _normal(g, shape, dtype), _normal(g, shape, dtype)
    elif kind == "latent":
        R, rank, q_rank = case["rot"], case["kv_rank"], case["q_rank"]
        out["weights"] = {"dq": w(q_rank, case["hidden"]), "dq.norm": 1 + _normal(g, (q_rank,), torch.float32, 0.01),
                          "uq": w(H * (D + R), q_rank), "dkv": w(rank + R, case["hidden"]),
                          "dkv.norm": 1 + _normal(g, (rank,), torch.float32, 0.01), "uk": w(H * D, rank), "uv": w(H * D, rank),
                          "o": w(case["hidden"], H * D)}
        out["table"], pages = _pages(g, contexts, PAGE)
        out["keys"] = _normal(g, (pages, 1, 1, PAGE, rank + R), dtype)
    else:
        V, hidden = case["vdim"], case["hidden"]
        matrices = _normal(g, (len(fed), H, D, V), torch.float32, 0.05)                # prompts go on from an earlier portion
        if kind == "recurrence":
            weights = {"q": w(H * D, hidden), "k": w(H * D, hidden), "v": w(H * V, hidden), "g": w(H * V, hidden), "o": w(hidden, H * V)}
            if case["decay"] == "channel_logits":
                weights.update({"a1": w(DECAY_RANK, hidden), "a2": w(H * D, DECAY_RANK, std=0.2), "a2.b": w(H * D),
                                "norm": 1 + _normal(g, (V,), torch.float32, 0.01)})
            out["state"] = matrices.reshape(len(fed), -1)
        else:
            G = case["kv_heads"]
            C = 2 * G * D + H * V
            weights = {"q": w(G * D, hidden), "k": w(G * D, hidden), "v": w(H * V, hidden), "b": w(H, hidden), "o": w(hidden, H * V),
                       "q.conv": w(G * D, TAPS, std=0.4), "k.conv": w(G * D, TAPS, std=0.4), "v.conv": w(H * V, TAPS, std=0.4),
                       "norm": 1 + _normal(g, (V,), torch.float32, 0.01)}
            rows = H if case["scope"] == "head" else H * D
            step = torch.exp(_uniform(g, (rows,), math.log(1e-3), math.log(1e-1)))     # decays from slow to fast, as trained ones spread
            weights["dt_bias"] = step + torch.log(-torch.expm1(-step))
            weights["A_log"] = torch.log(_uniform(g, (H,), 1.0, 16.0))
            if case["scope"] == "head":
                weights.update({"a": w(H, hidden), "g": w(H * V, hidden)})
            else:
                weights.update({"a1": w(DECAY_RANK, hidden), "a2": w(H * D, DECAY_RANK, std=0.2), "g1": w(GATE_RANK, hidden),
                                "g2": w(H * V, GATE_RANK, std=0.2)})
            taps = _normal(g, (len(fed), (TAPS - 1) * C), torch.float32, 0.9)
            out["state"] = torch.cat([matrices.reshape(len(fed), -1), taps], dim=1)
        out["weights"] = weights
    return out


# ----------------------------------------------------------------------------------------------- what a program holds, and the call
def _spec(case):
    kind, hidden = case["kind"], case["hidden"]
    if kind == "attention":
        rotary = RotarySpec(head_dim=case["dim"], theta=THETA, max_positions=16384, scaling=Llama3Scaling(32.0, 1.0, 4.0, 8192))
        return "mixer", AttentionSpec(hidden_size=hidden, num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=case["dim"],
                                      scale=case["dim"] ** -0.5, position=rotary)
    if kind == "ffn":
        return "feed_forward", GatedMLPSpec(hidden_size=hidden, intermediate_size=case["ff"])
    if kind == "experts":
        def expert(ff):
            return GatedMLPSpec(hidden_size=hidden, intermediate_size=ff, activation="clamped_swish", limit=SWISH_LIMIT, alpha=SWISH_ALPHA,
                                tensor_names=("gate", "up", "down"))
        return "feed_forward", RoutedExpertsSpec(hidden_size=hidden, num_experts=case["experts"], top=case["top"],
                                                 expert=expert(case["expert_ff"]), shared=expert(case["shared_ff"]))
    dim = case["dim"]
    if kind == "latent":
        return "mixer", LatentAttentionSpec(hidden_size=hidden, num_heads=case["heads"], head_dim=dim, rot_dim=case["rot"], value_dim=dim,
                                            q_rank=case["q_rank"], kv_rank=case["kv_rank"], scale=(dim + case["rot"]) ** -0.5,
                                            window=case["window"], norm_eps=NORM_EPS, position=InlineRotarySpec(dims=case["rot"]))
    if kind == "recurrence":
        sizes = dict(hidden_size=hidden, num_heads=case["heads"], key_dim=dim, value_dim=case["vdim"], out_norm_eps=NORM_EPS)
        if case["decay"] == "channel_logits":
            return "mixer", LinearRecurrenceSpec(q_scale=dim ** -0.5, decay="channel_logits", decay_rank=DECAY_RANK, tau=TAU, **sizes)
        return "mixer", LinearRecurrenceSpec(k_scale=dim ** -0.5, decay="head", head_decays=_head_decays(case),
                                             position=InlineRotarySpec(dims=dim), out_norm_weight=False, **sizes)
    head = case["scope"] == "head"
    return "mixer", GatedDeltaRuleSpec(hidden_size=hidden, num_heads=case["heads"], num_kv_heads=case["kv_heads"], key_dim=dim,
                                       value_dim=case["vdim"], conv_taps=TAPS, q_scale=dim ** -0.5, unit_eps=UNIT_EPS, out_norm_eps=NORM_EPS,
                                       decay_rank=0 if head else DECAY_RANK, gate_rank=0 if head else GATE_RANK,
                                       decay_scope=case["scope"], gate="silu" if head else "low_rank_sigmoid")


def _head_decays(case) -> tuple[float, ...]:
    return tuple(1.0 - 2.0 ** (-5 - i % 4) for i in range(case["heads"]))


def _i32(values) -> torch.Tensor:
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _context(fed: list[int], cached: list[int]) -> StepContext:
    """The step's index data as the step function packs it."""
    n = len(fed)
    cu_q = [0]
    for k in fed:
        cu_q.append(cu_q[-1] + k)
    ctx_lens = [a + b for a, b in zip(fed, cached)]
    ctx = StepContext(None, cu_q[-1], n, HostView(list(range(n)), cu_q, list(cached), ctx_lens, list(range(n))))
    ctx.positions = _i32([p for k, c in zip(fed, cached) for p in range(c, c + k)])
    ctx.seq_of_token = _i32([s for s, k in enumerate(fed) for _ in range(k)])
    ctx.cu_q, ctx.ctx_lens, ctx.state_slots = _i32(cu_q), _i32(ctx_lens), _i32(list(range(n)))
    ctx.prefill_seqs = _i32([s for s, k in enumerate(fed) if k > 1])
    return ctx


def prepare(case, seed) -> dict:
    inputs = _inputs(case, seed)
    rt = Runtime(dtype=DTYPES[case.get("dtype", "bf16")], device=torch.device(DEV, torch.cuda.current_device()), ops=get_ops())
    if case["kind"] == "step":
        model = DecoderModel(inputs["spec"], inputs["weights"], rt)
        layout = plan_layout(model.cache_needs(), PAGE)
        storage = DeviceCacheStorage(layout, inputs["pages"], rt.dtype, rt.device, rt.ops)
        manager = CacheManager(layout, inputs["pages"], storage, caching=False)
        runner = StepRunner(model, manager, storage, max_decode_batch=64)
        entries = []
        for i, token in enumerate(inputs["tokens"]):                    # requests whose contexts are in the cache already
            assert manager.admit(i, [0] * case["context"])
            manager.commit(i, case["context"])
            manager.extend(i, [token])
            held = case["context"] // PAGE + 1                           # a fresh pool hands its pages out in order
            assert manager.block_table(i) == list(range(i * held, (i + 1) * held))
            entries.append(StepEntry(i, [token], [0]))
        storage.k_pools[0].copy_(inputs["keys"])
        storage.v_pools[0].copy_(inputs["values"])
        return dict(runner=runner, entries=entries)
    role, spec = _spec(case)
    part = part_class(role, spec)(spec, inputs["weights"], rt)
    if role == "feed_forward":
        return dict(part=part, x=inputs["x"], ctx=_context([inputs["x"].shape[0]], [0]))
    ctx = _context(inputs["fed"], inputs["cached"])
    if "state" in inputs:
        state = inputs["state"].contiguous().view(torch.uint8)
        binding = EntryBinding(None, None, 0, 0, PAGE, 0, group=-1, state=state, state_slots=ctx.state_slots)
        return dict(part=part, x=inputs["x"], ctx=ctx, binding=binding, kept=[state.view(torch.float32)])
    keys, values, table = inputs["keys"], inputs.get("values"), inputs["table"]
    entry = keys[0].numel()
    binding = EntryBinding(keys, values, entry, 0, PAGE, keys.shape[0], table, table.shape[1])
    return dict(part=part, x=inputs["x"], ctx=ctx, binding=binding, kept=[t for t in (keys, values) if t is not None])


@torch.inference_mode()
def run(state):
    if "runner" in state:
        return state["runner"].step(state["entries"])                   # float32 logits
    if "binding" not in state:
        return state["part"].forward(state["x"], state["ctx"])
    y = state["part"].forward(state["x"], state["ctx"], state["binding"])
    return [y, *state["kept"]]                                          # the layer's output and the cache or state it has moved on


# ------------------------------------------------------------------------------------------------------- bytes and operations
def work(case) -> dict:
    kind = case["kind"]
    size = DTYPES[case.get("dtype", "bf16")].itemsize
    if kind == "step":
        n, ctx, c = case["requests"], case["context"], LLAMA_1B
        h, i, layers, v = c["hidden_size"], c["intermediate_size"], c["num_hidden_layers"], c["vocab_size"]
        weights = layers * (h * 3072 + 2048 * h + 3 * i * h) + v * h
        return {"bytes": 2 * weights + n * (ctx + 1) * layers * 2 * 512 * 2 + 4 * n * v,
                "flops": 2.0 * n * weights + 4.0 * n * layers * 2048 * (ctx + 1)}
    if kind == "ffn":
        weights = 3 * case["hidden"] * case["ff"]
        return {"bytes": size * (weights + 2 * case["rows"] * case["hidden"]), "flops": 2.0 * case["rows"] * weights}
    if kind == "experts":
        t, h = case["tokens"], case["hidden"]
        used = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** t)        # experts some token chooses, on average
        one, shared = 3 * h * case["expert_ff"], 3 * h * case["shared_ff"]
        return {"bytes": 2 * (used * one + shared + case["experts"] * h + 2 * t * h),
                "flops": 2.0 * t * (case["top"] * one + shared + case["experts"] * h)}
    fed, cached = _lengths(case)
    T, h, H, D = sum(fed), case["hidden"], case["heads"], case["dim"]
    if kind == "attention":
        kv = case["kv_heads"] * D
        weights = h * (H * D + 2 * kv) + H * D * h
        pairs = sum(n * (c + (n + 1) / 2) for n, c in zip(fed, cached))
        return {"bytes": size * (weights + 2 * T * h + 2 * kv * (2 * T + sum(cached))), "flops": 2.0 * T * weights + 4.0 * H * D * pairs}
    if kind == "latent":
        R, rank, q_rank, window = case["rot"], case["kv_rank"], case["q_rank"], case["window"]
        weights = h * (q_rank + rank + R) + q_rank * H * (D + R) + 2 * H * D * rank + H * D * h
        keys = [min(window, c + i + 1) if window else c + i + 1 for n, c in zip(fed, cached) for i in range(n)]
        read = sum(min(c, window - 1) if window else c for c in cached)
        # the scores and sums of heads of their own keys and values, the smallest form of this attention over a prompt
        return {"bytes": 2 * (weights + 2 * T * h + (rank + R) * (2 * T + read)), "flops": 2.0 * T * weights + 2.0 * H * (2 * D + R) * sum(keys)}
    V = case["vdim"]
    if kind == "recurrence":
        weights = h * (2 * H * D + 2 * H * V) + H * V * h + (DECAY_RANK * (h + H * D) if case["decay"] == "channel_logits" else 0)
        state = H * D * V
        ops = 5.0
    else:
        G = case["kv_heads"]
        low = H * h + h * H * V if case["scope"] == "head" else DECAY_RANK * (h + H * D) + GATE_RANK * (h + H * V)
        weights = h * (2 * G * D + H * V + H) + H * V * h + low
        state = H * D * V + (TAPS - 1) * (2 * G * D + H * V)
        ops = 7.0
    return {"bytes": 2 * (weights + 2 * T * h) + 2 * 4 * len(fed) * state, "flops": 2.0 * T * weights + ops * T * H * D * V}


def tolerance(case):
    # measured against `exact`: layers 0.0035 to 0.0057 in bfloat16 and 2e-6 in 32 bits; the sixteen layers of a whole step,
    # whose roundings travel through all that follow, 0.028 to 0.033; about four times that between two correct forms
    kind = case["kind"]
    if case.get("dtype") == "f32":
        return {"rel": 1e-5}
    return {"rel": {"step": 1e-1, "attention": 2e-2, "ffn": 2e-2, "recurrence": 2e-2, "delta": 2e-2, "latent": 2e-2, "experts": 2e-2}[kind]}


# ------------------------------------------------------------------------------------------------------------- the same in 64 bits
def _f64(t: torch.Tensor) -> torch.Tensor:
    return t.to(torch.float64)


def _rotation(positions, frequencies) -> tuple[torch.Tensor, torch.Tensor]:
    """Cosines and sines of the model's angles, which are float32 products."""
    angle = (positions.to(torch.float32)[:, None] * frequencies[None, :]).to(torch.float64)
    return angle.cos(), angle.sin()


def _rotate(x, cos, sin):
    """x [T, heads, 2 n], channel i with channel i + n."""
    a, b = x.chunk(2, dim=-1)
    return torch.cat([a * cos[:, None] - b * sin[:, None], b * cos[:, None] + a * sin[:, None]], dim=-1)


def _llama_frequencies(dim: int) -> torch.Tensor:
    f = 1.0 / (THETA ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim))
    wave = 2 * math.pi / f
    factor, low, high, window = 32.0, 1.0, 4.0, 8192
    slow = torch.where(wave > window / low, f / factor, f)
    s = (window / wave - low) / (high - low)
    blend = (1 - s) * slow / factor + s * slow
    return torch.where((wave >= window / high) & (wave <= window / low), blend, slow).to(DEV)


def _frequencies(dims: int, base: float = 10000.0) -> torch.Tensor:
    return (base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64) / dims)).to(torch.float32).to(DEV)


def _slots(table: torch.Tensor, row: int, n: int, start: int = 0):
    at = torch.arange(start, start + n, device=DEV)
    return table[row, at // PAGE].long(), at % PAGE


def _softmax_attention(q, k, v, first: int, scale: float, window: int = 0):
    """q [T, H, D] at positions first.., k [n, G, D], v [n, G, V]: [T, H, V], a head at a time."""
    T, H, n, group = q.shape[0], q.shape[1], k.shape[0], q.shape[1] // k.shape[1]
    i = torch.arange(first, first + T, device=DEV)[:, None]
    j = torch.arange(n, device=DEV)[None, :]
    hidden = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // group].t() * scale).masked_fill(hidden, -math.inf)
        out.append(torch.softmax(s, dim=-1) @ v[:, h // group])
    return torch.stack(out, dim=1)


def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


@torch.inference_mode()
def exact(case, seed):
    a = _inputs(case, seed)
    if case["kind"] == "step":
        return _exact_step(case, a)
    w = {k: _f64(t) for k, t in a["weights"].items()}
    x = _f64(a["x"])
    if case["kind"] == "ffn":
        return (_silu(x @ w["gate_proj.weight"].t()) * (x @ w["up_proj.weight"].t())) @ w["down_proj.weight"].t()
    if case["kind"] == "experts":
        return _exact_experts(case, w, x)
    return {"attention": _exact_attention, "latent": _exact_latent, "recurrence": _exact_recurrence,
            "delta": _exact_delta}[case["kind"]](case, a, w, x)


def _exact_step(case, a):
    w, n, context = a["weights"], case["requests"], case["context"]
    per, held = -(-context // PAGE), context // PAGE + 1
    x = _f64(w["model.embed_tokens.weight"][torch.tensor(a["tokens"], device=DEV)])
    cos, sin = _rotation(torch.full((n,), context, device=DEV), _llama_frequencies(64))
    eps = LLAMA_1B["rms_norm_eps"]
    for l in range(LLAMA_1B["num_hidden_layers"]):
        m = {k: _f64(t) for k, t in w.items() if k.startswith(f"model.layers.{l}.")}
        p = f"model.layers.{l}."
        h = _rms(x, eps) * m[p + "input_layernorm.weight"]
        q = _rotate((h @ m[p + "self_attn.q_proj.weight"].t()).view(n, 32, 64), cos, sin)
        k = _rotate((h @ m[p + "self_attn.k_proj.weight"].t()).view(n, 8, 64), cos, sin)
        v = (h @ m[p + "self_attn.v_proj.weight"].t()).view(n, 8, 64)
        o = []
        for s in range(n):
            pages = torch.arange(s * held, s * held + per, device=DEV)
            ks = _f64(a["keys"][pages, l]).transpose(1, 2).reshape(-1, 8, 64)[:context]
            vs = _f64(a["values"][pages, l]).transpose(1, 2).reshape(-1, 8, 64)[:context]
            o.append(_softmax_attention(q[s:s + 1], torch.cat([ks, k[s:s + 1]]), torch.cat([vs, v[s:s + 1]]), context, 0.125))
        x = x + torch.cat(o).reshape(n, -1) @ m[p + "self_attn.o_proj.weight"].t()
        h = _rms(x, eps) * m[p + "post_attention_layernorm.weight"]
        x = x + (_silu(h @ m[p + "mlp.gate_proj.weight"].t()) * (h @ m[p + "mlp.up_proj.weight"].t())) @ m[p + "mlp.down_proj.weight"].t()
    h = _rms(x, eps) * _f64(w["model.norm.weight"])
    return torch.cat([h @ _f64(part).t() for part in w["model.embed_tokens.weight"].split(16384)], dim=1)


def _exact_attention(case, a, w, x):
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    T = x.shape[0]
    positions = torch.cat([torch.arange(c, c + n, device=DEV) for n, c in zip(a["fed"], a["cached"])])
    cos, sin = _rotation(positions, _llama_frequencies(D))
    q = _rotate((x @ w["q_proj.weight"].t()).view(T, H, D), cos, sin)
    k = _rotate((x @ w["k_proj.weight"].t()).view(T, G, D), cos, sin)
    v = (x @ w["v_proj.weight"].t()).view(T, G, D)
    keys, values = _f64(a["keys"]), _f64(a["values"])
    out, at = [], 0
    for s, (n, c) in enumerate(zip(a["fed"], a["cached"])):
        page, slot = _slots(a["table"], s, n, c)
        keys[page, 0, :, slot], values[page, 0, :, slot] = k[at:at + n], v[at:at + n]
        page, slot = _slots(a["table"], s, c + n)
        out.append(_softmax_attention(q[at:at + n], keys[page, 0, :, slot], values[page, 0, :, slot], c, D ** -0.5))
        at += n
    return [torch.cat(out).reshape(T, H * D) @ w["o_proj.weight"].t(), keys, values]


def _exact_latent(case, a, w, x):
    H, D, R, rank = case["heads"], case["dim"], case["rot"], case["kv_rank"]
    T = x.shape[0]
    positions = torch.cat([torch.arange(c, c + n, device=DEV) for n, c in zip(a["fed"], a["cached"])])
    cos, sin = _rotation(positions, _frequencies(R))
    c_q = _rms(x @ w["dq"].t(), NORM_EPS) * w["dq.norm"]
    q = (c_q @ w["uq"].t()).view(T, H, D + R)
    q = torch.cat([q[..., :D], _rotate(q[..., D:], cos, sin)], dim=-1)
    y = x @ w["dkv"].t()
    row = torch.cat([_rms(y[:, :rank], NORM_EPS) * w["dkv.norm"], _rotate(y[:, None, rank:], cos, sin)[:, 0]], dim=-1)
    keys = _f64(a["keys"])
    out, at = [], 0
    for s, (n, c) in enumerate(zip(a["fed"], a["cached"])):
        page, slot = _slots(a["table"], s, n, c)
        keys[page, 0, 0, slot] = row[at:at + n]
        page, slot = _slots(a["table"], s, c + n)
        rows = keys[page, 0, 0, slot]
        latent, rotated = rows[:, :rank], rows[:, None, rank:].expand(-1, H, R)
        k = torch.cat([(latent @ w["uk"].t()).view(-1, H, D), rotated], dim=-1)
        v = (latent @ w["uv"].t()).view(-1, H, D)
        out.append(_softmax_attention(q[at:at + n], k, v, c, (D + R) ** -0.5, case["window"]))
        at += n
    return [torch.cat(out).reshape(T, H * D) @ w["o"].t(), keys]


def _exact_experts(case, w, x):
    def act(g, u):
        g, u = g.clamp(max=SWISH_LIMIT), u.clamp(-SWISH_LIMIT, SWISH_LIMIT)
        return g * torch.sigmoid(SWISH_ALPHA * g) * (u + 1)

    def expert(p, h):
        return act(h @ w[p + "gate"].t(), h @ w[p + "up"].t()) @ w[p + "down"].t()

    z, chosen = (x @ w["router"].t() + w["router.b"]).topk(case["top"], dim=-1)
    share = torch.softmax(z, dim=-1)
    out = expert("shared.", x)
    for e in range(case["experts"]):
        t, c = (chosen == e).nonzero(as_tuple=True)
        if t.numel():
            out.index_add_(0, t, expert(f"e{e}.", x[t]) * share[t, c][:, None])
    return out


def _exact_recurrence(case, a, w, x):
    H, D, V, T = case["heads"], case["dim"], case["vdim"], x.shape[0]
    q, k, v = (x @ w["q"].t()).view(T, H, D), (x @ w["k"].t()).view(T, H, D), (x @ w["v"].t()).view(T, H, V)
    if case["decay"] == "channel_logits":
        z = (x @ w["a1"].t()) @ w["a2"].t() + w["a2.b"]
        decay = torch.exp(torch.nn.functional.logsigmoid(z) / TAU).view(T, H, D)
        q = q * D ** -0.5
    else:
        decay = torch.tensor(_head_decays(case), dtype=torch.float32, device=DEV).to(torch.float64)[None, :, None].expand(T, H, D)
        positions = torch.cat([torch.arange(n, device=DEV) for n in a["fed"]])
        cos, sin = _rotation(positions, _frequencies(D))
        q, k = _rotate(q, cos, sin), _rotate(k, cos, sin) * D ** -0.5
    state = _f64(a["state"]).view(-1, H, D, V)
    o, at = torch.empty_like(v), 0
    for s, n in enumerate(a["fed"]):
        S = state[s].clone()
        for t in range(at, at + n):
            S = S * decay[t][..., None] + k[t][..., None] * v[t][:, None, :]
            o[t] = (S * q[t][..., None]).sum(1)
        state[s], at = S, at + n
    o = _rms(o, NORM_EPS)
    if "norm" in w:
        o = o * w["norm"]
    return [(o.reshape(T, H * V) * _silu(x @ w["g"].t())) @ w["o"].t(), state.reshape(len(a["fed"]), -1)]


def _exact_delta(case, a, w, x):
    H, G, D, V, T = case["heads"], case["kv_heads"], case["dim"], case["vdim"], x.shape[0]
    C = 2 * G * D + H * V
    raw = torch.cat([x @ w["q"].t(), x @ w["k"].t(), x @ w["v"].t()], dim=-1)
    taps = torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]], dim=0)                    # [C, taps]
    state = _f64(a["state"])
    matrices, carried = state[:, :H * D * V].reshape(-1, H, D, V).clone(), state[:, H * D * V:].reshape(-1, TAPS - 1, C).clone()
    beta = torch.sigmoid(x @ w["b"].t())
    rate = torch.exp(w["A_log"])
    if case["scope"] == "head":
        z = torch.nn.functional.softplus(x @ w["a"].t() + w["dt_bias"])
        decay = torch.exp(-rate * z)[..., None].expand(T, H, D)
    else:
        z = torch.nn.functional.softplus((x @ w["a1"].t()) @ w["a2"].t() + w["dt_bias"]).view(T, H, D)
        decay = torch.exp(-rate[None, :, None] * z)
    o, at = torch.empty((T, H, V), dtype=torch.float64, device=DEV), 0
    for s, n in enumerate(a["fed"]):
        line = torch.cat([carried[s], raw[at:at + n]])
        conv = _silu(sum(line[i:i + n] * taps[:, i] for i in range(TAPS)))
        carried[s] = line[-(TAPS - 1):]
        q, k = conv[:, :G * D].view(n, G, D), conv[:, G * D:2 * G * D].view(n, G, D)
        v = conv[:, 2 * G * D:].view(n, H, V)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + UNIT_EPS) * D ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + UNIT_EPS)
        q, k = q.repeat_interleave(H // G, dim=1), k.repeat_interleave(H // G, dim=1)
        S = matrices[s]
        for t in range(n):
            S = S * decay[at + t][..., None]
            u = beta[at + t][:, None] * (v[t] - (S * k[t][..., None]).sum(1))
            S = S + k[t][..., None] * u[:, None, :]
            o[at + t] = (S * q[t][..., None]).sum(1)
        matrices[s], at = S, at + n
    o = (_rms(o, NORM_EPS) * w["norm"]).reshape(T, H * V)
    gate = _silu(x @ w["g"].t()) if case["scope"] == "head" else torch.sigmoid((x @ w["g1"].t()) @ w["g2"].t())
    return [(o * gate) @ w["o"].t(), torch.cat([matrices.reshape(len(a["fed"]), -1), carried.reshape(len(a["fed"]), -1)], dim=1)]
