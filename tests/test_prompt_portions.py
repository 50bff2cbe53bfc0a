"""Kernels that only prompt portions reach (tiles of sixteen tokens, runs of the convolution, head norms by wide loads), at their edges."""

from __future__ import annotations

import pytest
import torch

from gpu_util import i32, make_ctx
from tinyserve_llm_b200.cache.storage import EntryBinding
from tinyserve_llm_b200.ops import KernelError, get_ops
from tinyserve_llm_b200.parts.delta_rule import CHANNEL_TILE_TOKENS
from tinyserve_llm_b200.parts.recurrence import TILE_TOKENS

pytestmark = pytest.mark.gpu

LENS = [1, 2, 15, 16, 17, 33, 1, 75]                    # single tokens go to the scan, beside tiles that are full, short and one over


def _step(state, lens=LENS):
    ctx = make_ctx(lens, [n + 5 * s for s, n in enumerate(lens)])
    ctx.prefill_seqs = i32([s for s, n in enumerate(lens) if n > 1])
    rows = state.shape[0]
    return ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state.view(torch.uint8).view(rows, -1), state_slots=i32([rows - 1 - s for s in range(len(lens))]))


def _close_to_64_bits(got, want, heads):
    """By head: the worst row and the median of the norm of the difference.  A term of either path carries about 2^-21 of itself; the
    worst rows are those whose terms cancel."""
    got, want = (t.reshape(t.shape[0], heads, -1) for t in (got.double().cpu(), want))
    err = (got - want).norm(dim=-1) / want.norm(dim=-1).clamp_min(1e-30)
    assert float(err.max()) < 2e-4 and float(err.median()) < 5e-6, f"worst {float(err.max()):.2e}, median {float(err.median()):.2e}"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("decays", ["channel", "head", "gone"])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (100, 52), (128, 40), (256, 129)])
def test_plain_recurrence_of_portions(dim, vdim, decays, dtype):
    ops, H, tau = get_ops(), 3, 4.0
    g = torch.Generator().manual_seed(dim + vdim)
    T = sum(LENS)
    y = (torch.randn(T, H * (2 * dim + vdim) + 4, generator=g) * 0.5).to(dtype)
    z = torch.randn(T, H * dim, generator=g) + 5
    if decays == "gone":                                 # decays that are zero in float32, beside ones near one
        z[:, ::3] = -1e4
    per_head = torch.tensor([0.999, 0.7, 1e-30])
    state = torch.randn(len(LENS) + 3, H * dim * vdim, generator=g)
    dev, yd = state.cuda(), y.cuda()
    ctx, binding = _step(dev)
    cuts = (0, H * dim, 2 * H * dim, H * (2 * dim + vdim))
    q, k, v = (yd[:, a:b] for a, b in zip(cuts, cuts[1:]))
    logits = dict(z=None, bias=None, head_decays=per_head.cuda()) if decays == "head" else dict(z=z.cuda(), bias=None, head_decays=None)
    before = ops.calls.get("ts_plain_tiles", 0)
    got = ops.linear_recurrence(q, k, v, ctx, binding, heads=H, dim=dim, vdim=vdim, inv_tau=1 / tau, q_scale=0.7, k_scale=1.3, **logits)
    assert ops.calls.get("ts_plain_tiles", 0) == before + 1
    qh, kh, vh = (y[:, a:b].double().view(T, H, -1) for a, b in zip(cuts, cuts[1:]))
    a = per_head.double()[None, :, None].expand(T, H, dim) if decays == "head" else torch.sigmoid(z.double()).pow(1 / tau).view(T, H, dim)

    def walk(q, k, v, left):
        out, at = torch.empty(T, H, vdim, dtype=torch.float64), 0
        for s, n in enumerate(LENS):
            S = left[len(left) - 1 - s]
            for t in range(at, at + n):
                S.mul_(a[t][:, :, None]).add_(1.3 * k[t][:, :, None] * v[t][:, None, :])
                out[t] = 0.7 * torch.einsum("hdv,hd->hv", S, q[t])
            at += n
        return out, left

    start = state.double().view(-1, H, dim, vdim)
    want, left = walk(qh, kh, vh, start.clone())
    size, left_size = walk(qh.abs(), kh.abs(), vh.abs(), start.abs())                   # what the terms amount to: a head without memory is q . k, which cancels
    # a product of split operands is within 2^-21, a decay product over up to 75 steps within 75 2^-23; twice their sum
    for mine, true, terms in ((got, want, size), (dev, left, left_size)):
        mine, true, terms = (t.double().cpu().reshape(-1, H, true[0, 0].numel()) for t in (mine, true, terms))
        worst = float(((mine - true).norm(dim=-1) / terms.norm(dim=-1).clamp_min(1e-30)).max())
        assert worst < 2e-5, f"{worst:.2e} of the terms"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("decay", [-6.0, 0.0, 30.0])
@pytest.mark.parametrize("dim,vdim,heads,kv_heads", [(64, 64, 2, 1), (100, 52, 3, 3), (128, 128, 2, 1), (256, 33, 2, 2)])
def test_channel_decayed_delta_rule_of_portions(dim, vdim, heads, kv_heads, decay, dtype):
    """From decays near one to decays that are zero in float32, with keys that repeat (the delta rule's corrections are then large)."""
    ops, H, G = get_ops(), heads, kv_heads
    g = torch.Generator().manual_seed(dim + vdim)
    T, C = sum(LENS), 2 * kv_heads * dim + heads * vdim
    conv = torch.randn(T, C, generator=g)
    conv[1::2, G * dim:2 * G * dim] = conv[0:T - 1:2, G * dim:2 * G * dim][:conv[1::2].shape[0]]
    z = torch.randn(T, H * dim, generator=g) + decay
    b = (torch.randn(T, H, generator=g) * 2).to(dtype)
    dt_bias, a_log = torch.randn(H * dim, generator=g) * 0.3, torch.randn(H, generator=g) * 0.5
    state = torch.randn(len(LENS) + 3, H * dim * vdim, generator=g)
    dev, cd = state.cuda(), conv.cuda()
    ctx, binding = _step(dev)
    sizes = dict(heads=H, kv_heads=G, dim=dim, unit_eps=1e-6, q_scale=0.25)
    parts = cd[:, :G * dim], cd[:, G * dim:2 * G * dim], cd[:, 2 * G * dim:]
    rest = z.cuda(), b.cuda(), dt_bias.cuda(), a_log.cuda()
    got = ops.channel_tiles(*parts, *rest, ctx, binding, vdim=vdim, **sizes)
    prepared, beta = ops.delta_prepare(parts[0], parts[1], rest[0], rest[2], rest[3], rest[1], **sizes)
    got = ops.recurrence_scan(prepared, parts[2], ctx, binding, heads=H, dim=dim, vdim=vdim, beta=beta, singles=True, out=got)
    q, k, a = (t.double().cpu().view(T, H, dim) for t in prepared)                      # as the token-by-token walk takes them
    bt, v = beta.double().cpu(), conv[:, 2 * G * dim:].double().view(T, H, vdim)
    want, left = torch.empty(T, H, vdim, dtype=torch.float64), state.double().view(-1, H, dim, vdim).clone()
    at = 0
    for s, n in enumerate(LENS):
        S = left[len(left) - 1 - s]
        for t in range(at, at + n):
            S.mul_(a[t][:, :, None])
            S.add_(k[t][:, :, None] * (bt[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None, :])
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        at += n
    _close_to_64_bits(got, want, H)
    _close_to_64_bits(dev, left.view(len(left), -1), H)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens,channels", [([256], 4), ([1, 2, 3, 4, 5, 250, 7], 516), ([300] + [1] * 13, 1032), ([8] * 33, 128)])
def test_convolution_by_runs_of_tokens_is_the_convolution(lens, channels, dtype):
    """The same bits from rows that wide loads take (runs of tokens) and from rows one element further (an element at a time)."""
    ops = get_ops()
    g = torch.Generator().manual_seed(channels)
    T = sum(lens)
    wide = torch.zeros(T, channels + 8, dtype=dtype, device="cuda")
    x = torch.randn(T, channels, generator=g).to(dtype).cuda()
    taps = torch.randn(channels, 4, generator=g).cuda()
    state = torch.randn(len(lens) + 3, 3 * channels, generator=g).cuda()
    results = []
    for offset in (0, 1):
        held = state.clone()
        ctx, binding = _step(held, lens)
        ctx.seq_of_token[-1] = -1 if lens[-1] == 1 else ctx.seq_of_token[-1]                # a padding row
        wide[:, offset:offset + channels] = x
        y = ops.short_conv_silu(wide[:, offset:offset + channels], taps, ctx, binding)
        results.append((y[:T - 1] if lens[-1] == 1 else y, held))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])
    n = lens[0]
    past = state[-1].view(3, channels).double()
    full = torch.cat([past, x[:n].double()])
    acc = sum(full[j:j + n] * taps[:, j].double() for j in range(4))
    torch.testing.assert_close(results[0][0][:n].double(), torch.nn.functional.silu(acc), atol=3e-6, rtol=3e-6)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,heads,vdim", [(1, 1, 128), (3, 3, 256), (33, 5, 128), (2, 1, 384)])
@pytest.mark.parametrize("kind,per_head", [("silu", False), ("sigmoid", True), ("silu", None)])
def test_head_norm_by_wide_loads(tokens, heads, vdim, kind, per_head, dtype):
    """Columns of wider tensors, on the loads' boundaries and beside them."""
    ops = get_ops()
    g = torch.Generator().manual_seed(vdim + tokens)
    n, eps = heads * vdim, 1e-5
    o = torch.randn(tokens, n, generator=g) * 3
    gate = torch.randn(tokens, n, generator=g).to(dtype)
    weight = None if per_head is None else 1 + torch.randn(n if per_head else vdim, generator=g) * 0.3
    oh = o.double().view(tokens, heads, vdim)
    w = 1.0 if weight is None else weight.double().view(-1, vdim)
    act = torch.nn.functional.silu if kind == "silu" else torch.sigmoid
    want = (oh / (oh.pow(2).mean(-1, keepdim=True) + eps).sqrt() * w).view(tokens, n) * act(gate.double()) * 0.5
    # one rounding to the type behind float32 steps
    tol = dict(atol=2e-6, rtol=4e-6) if dtype == torch.float32 else dict(atol=1e-6, rtol=2.0 ** -8)
    for offset in (0, 4, 1):
        wide, into = (torch.zeros(tokens, n + 8, dtype=dtype, device="cuda") for _ in range(2))
        wide[:, offset:offset + n] = gate.cuda()
        ops.head_norm_gate(o.cuda(), wide[:, offset:offset + n], None if weight is None else weight.cuda(), heads, vdim, eps, dtype, gate_kind=kind,
                           weight_per_head=bool(per_head), scale=0.5, out=into[:, offset:offset + n])
        torch.testing.assert_close(into[:, offset:offset + n].double().cpu(), want, **tol)
        into[:, offset:offset + n] = 0
        assert not into.any()


def _portion_of_mode(mode, plant):
    """One form of the recurrences over the portions of LENS: {input: value} planted in a token's inputs."""
    ops, H, G, D, V = get_ops(), 2, 1, 64, 64
    T = sum(LENS)
    g = torch.Generator().manual_seed(5)
    heads = G if mode in ("head", "channel") else H
    inputs = {"q": torch.randn(T, heads * D, generator=g), "k": torch.randn(T, heads * D, generator=g), "v": torch.randn(T, H * V, generator=g),
              "z": torch.randn(T, H * D, generator=g), "b": torch.randn(T, H, generator=g), "gates": torch.randn(T, 2 * H, generator=g)}
    for name, (token, column, value) in plant.items():
        inputs[name][token, column] = value
    x = {name: t.cuda() for name, t in inputs.items()}
    state = torch.randn(len(LENS), H * D * V, generator=g).cuda()
    ctx, binding = _step(state)
    sizes = dict(heads=H, kv_heads=G, dim=D, vdim=V, unit_eps=1e-6, q_scale=0.25)
    per_head, per_channel = torch.zeros(H).cuda(), torch.zeros(H * D).cuda()
    if mode == "plain":
        out = ops.linear_recurrence(x["q"], x["k"], x["v"], ctx, binding, heads=H, dim=D, vdim=V, z=x["z"], bias=None, head_decays=None, inv_tau=0.1,
                                    q_scale=0.25, k_scale=1.0)
    elif mode == "mixing":
        out = ops.mix_tiles(x["q"], x["k"], x["v"], x["z"], per_channel, per_channel + 0.5, ctx, binding, heads=H, dim=D)
    elif mode == "channel":
        out = ops.channel_tiles(x["q"], x["k"], x["v"], x["z"], x["b"], per_channel, per_head, ctx, binding, **sizes)
    else:
        out = ops.delta_tiles(x["q"], x["k"], x["v"], x["gates"], per_head, per_head, ctx, binding, **sizes)
    for s, n in enumerate(LENS):
        if n == 1:                                       # not written by the tiles
            out[sum(LENS[:s])] = 0
    return out.view(T, H, V).cpu()


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 3.401e38])
@pytest.mark.parametrize("mode,name", [(m, n) for m, names in (("plain", "qkvz"), ("mixing", "qkvz"), ("channel", "qkvzb"), ("head", ["q", "k", "v", "gates"])) for n in names])
def test_what_is_not_finite_reaches_no_earlier_token(mode, name, value):
    """A token in the middle of a tile, in the portion of 75 tokens: the rows before it and the other requests' keep their bits."""
    begin = sum(LENS[:-1])
    token = begin + 37
    clean, got = _portion_of_mode(mode, {}), _portion_of_mode(mode, {name: (token, 1, value)})
    assert torch.equal(got[:token], clean[:token])
    if name == "v":                                      # head 0, column 1, from the token on; everything else stands
        assert not torch.equal(got[token:, 0, 1], clean[token:, 0, 1])
        got[token:, 0, 1] = clean[token:, 0, 1]
        assert torch.equal(got, clean)
    elif name in "qk" and value != value:
        assert not torch.isfinite(got[token]).all()


@pytest.mark.parametrize("form,tokens,heads", [("channel", 70, 3), ("head", 70, 4), ("head", 400, 2), ("delta", 300, 3)])
def test_tiles_are_no_further_from_64_bits_than_the_walk(form, tokens, heads):
    """bfloat16 values, decays as trained models spread them: outputs and states of both ways against the same recurrence in 64 bits."""
    ops, H, D, V, T = get_ops(), heads, 128, 48, tokens
    g = torch.Generator().manual_seed(tokens)
    y = (torch.randn(T, H * (2 * D + V), generator=g) * 0.9).to(torch.bfloat16)
    z, state = torch.randn(T, H * D, generator=g) * 0.7, torch.randn(1, H * D * V, generator=g) * 0.05
    cuts = (0, H * D, 2 * H * D, H * (2 * D + V))
    q, k, v = (y[:, a:b] for a, b in zip(cuts, cuts[1:]))
    per_head = torch.tensor([1 - 2.0 ** (-5 - h) for h in range(H)])
    wide = lambda t: t.double().view(T, H, -1)
    if form == "delta":
        q, k, v = (torch.nn.functional.silu(t.float()) for t in (q, k, v))
        logits, rate, bias = torch.randn(T, H, generator=g), torch.linspace(0, 2.5, H), torch.linspace(-6, -2, H * D)
        qd, kd = (wide(t) / (wide(t).pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() for t in (q, k))
        qd, beta = qd * 0.25, torch.sigmoid(logits.double())
        a = torch.exp(-rate.double().exp()[:, None] * torch.nn.functional.softplus(wide(z) + bias.double().view(H, D)))
    else:
        qd, kd = wide(q) * 0.25, wide(k)
        a = per_head.double()[None, :, None].expand(T, H, D) if form == "head" else torch.sigmoid(wide(z)).pow(1 / 16)
    S, want = state.double().view(H, D, V).clone(), torch.empty(T, H, V, dtype=torch.float64)
    for t in range(T):
        S *= a[t][:, :, None]
        u = wide(v)[t] if form != "delta" else beta[t][:, None] * (wide(v)[t] - torch.einsum("hdv,hd->hv", S, kd[t]))
        S += kd[t][:, :, None] * u[:, None, :]
        want[t] = torch.einsum("hdv,hd->hv", S, qd[t])
    off = []
    for tiles in (True, False):
        held = state.cuda()
        ctx, binding = _step(held, [T])
        if form == "delta":
            parts, rest = [t.cuda() for t in (q, k, v)], [t.cuda() for t in (z, logits, bias, rate)]
            sizes = dict(heads=H, kv_heads=H, dim=D, unit_eps=1e-6, q_scale=0.25)
            if tiles:
                got = ops.channel_tiles(*parts, *rest, ctx, binding, vdim=V, **sizes)
            else:
                prepared, b = ops.delta_prepare(parts[0], parts[1], rest[0], rest[2], rest[3], rest[1], **sizes)
                got = ops.recurrence_scan(prepared, parts[2], ctx, binding, heads=H, dim=D, vdim=V, beta=b)
        else:
            if not tiles:
                ctx.prefill_seqs = None
            yd = y.cuda()
            got = ops.linear_recurrence(*(yd[:, i:j] for i, j in zip(cuts, cuts[1:])), ctx, binding, heads=H, dim=D, vdim=V, bias=None,
                                        z=z.cuda() if form == "channel" else None, head_decays=per_head.cuda() if form == "head" else None,
                                        inv_tau=1 / 16, q_scale=0.25, k_scale=1.0)
        off += [float((x.double().cpu().view(-1) - y64.reshape(-1)).norm() / y64.norm()) for x, y64 in ((got, want), (held, S))]
    assert off[0] <= off[2] and off[1] <= off[3], off


def _stretched(dim, vdim, T, plant=None, name="v"):
    """bfloat16 portions of T, 1 and 130 tokens by stretches: (output, states, what 64 bits give for both)."""
    ops, H, lens = get_ops(), 3, [T, 1, 130]
    g = torch.Generator().manual_seed(dim + vdim)
    n = sum(lens)
    y = (torch.randn(n, H * (2 * dim + vdim) + 4, generator=g) * 0.5).to(torch.bfloat16)
    z, state = torch.randn(n, H * dim, generator=g) + 3, torch.randn(len(lens) + 3, H * dim * vdim, generator=g)
    cuts = (0, H * dim, 2 * H * dim, H * (2 * dim + vdim))
    if plant is not None:
        row, column, value = plant
        (z if name == "z" else y)[row, {"q": 0, "k": cuts[1], "v": cuts[2], "z": 0}[name] + column] = value
    dev, yd = state.cuda(), y.cuda()
    ctx, binding = _step(dev, lens)
    before = ops.calls.get("ts_plain_tiles", 0)
    got = ops.linear_recurrence(*(yd[:, a:b] for a, b in zip(cuts, cuts[1:])), ctx, binding, heads=H, dim=dim, vdim=vdim, z=z.cuda(), bias=None, head_decays=None,
                                inv_tau=1 / 16, q_scale=0.25, k_scale=1.0)
    assert ops.calls.get("ts_plain_tiles", 0) == before + 1
    q, k, v = (y[:, a:b].double().view(n, H, -1) for a, b in zip(cuts, cuts[1:]))
    a = torch.sigmoid(z.double()).pow(1 / 16).view(n, H, dim)
    want, left, at = torch.empty(n, H, vdim, dtype=torch.float64), state.double().view(-1, H, dim, vdim).clone(), 0
    for s, m in enumerate(lens if plant is None else []):
        S = left[len(left) - 1 - s]
        for t in range(at, at + m):
            S.mul_(a[t][:, :, None]).add_(k[t][:, :, None] * v[t][:, None, :])
            want[t] = 0.25 * torch.einsum("hdv,hd->hv", S, q[t])
        at += m
    return got.cpu(), dev.cpu(), want, left


@pytest.mark.parametrize("dim,vdim,T", [(64, 64, 129), (100, 129, 300), (128, 72, 257), (256, 33, 128), (36, 8, 513)])
def test_plain_recurrence_by_stretches(dim, vdim, T):
    """Portions around one stretch of 128 tokens and over several, rows and columns that fill their blocks and do not."""
    got, states, want, left = _stretched(dim, vdim, T)
    # as test_plain_recurrence_of_portions, over T tokens: a product within 2^-21, decays within sqrt(T) 2^-24 once roundings go both ways
    for mine, true in ((got, want), (states, left)):
        mine = mine.double().reshape(true.shape)
        assert float((mine - true).norm() / true.norm()) < 2.0 ** -21 + T ** 0.5 * 2.0 ** -24


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_a_value_that_is_not_finite_stays_in_its_column_by_stretches(value):
    (clean, *_), (got, *_) = _stretched(64, 40, 300), _stretched(64, 40, 300, (201, 2 * 40 + 17, value))
    assert torch.equal(got[:201], clean[:201]) and not torch.isfinite(got[201:300, 2 * 40 + 17]).any()
    got[201:300, 2 * 40 + 17] = clean[201:300, 2 * 40 + 17]
    assert torch.equal(got, clean)


@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 3.38e38])
@pytest.mark.parametrize("name", ["q", "k", "z"])
def test_what_is_not_finite_stays_with_its_head_and_later_tokens_by_stretches(name, value):
    """In the middle of a tile, a stretch behind it and one before: earlier tokens, other heads and other requests keep their bits, states too."""
    dim, vdim, token = 64, 40, 201
    (clean, states, *_), (got, left, *_) = _stretched(dim, vdim, 300), _stretched(dim, vdim, 300, (token, dim + 5, value), name)
    assert torch.equal(got[:token], clean[:token]) and torch.equal(got[300:], clean[300:])
    mine = slice(vdim, 2 * vdim)                         # the second head's outputs
    if name in "qk" and value != 3.38e38:
        assert not torch.isfinite(got[token, mine]).any()
    end = token + 1 if name == "q" else 300
    got[token:end, mine] = clean[token:end, mine]
    assert torch.equal(got, clean)
    if name != "q":                                      # the state of that request's head, in the planted channel's row
        row = states[-1].view(3, dim, vdim)[1, 5].clone()
        left[-1].view(3, dim, vdim)[1, 5] = row
    assert torch.equal(left, states)


def _recurrence_part(kind, dtype):
    from tinyserve_llm_b200.config.spec import GatedDeltaRuleSpec, LinearRecurrenceSpec
    from tinyserve_llm_b200.parts.base import Runtime, part_class
    g = torch.Generator().manual_seed(3)
    w = lambda *shape: torch.randn(shape, generator=g) * 0.05
    if kind == "plain":
        spec = LinearRecurrenceSpec(q_scale=0.125, decay="channel_logits", decay_rank=16, tau=16.0, hidden_size=128, num_heads=2, key_dim=64, value_dim=128,
                                    out_norm_eps=1e-6)
        tensors = {"q": w(128, 128), "k": w(128, 128), "v": w(256, 128), "g": w(256, 128), "o": w(128, 256), "a1": w(16, 128), "a2": w(128, 16) * 4,
                   "a2.b": w(128), "norm": 1 + w(128)}
    else:
        spec = GatedDeltaRuleSpec(hidden_size=128, num_heads=2, num_kv_heads=1, key_dim=64, value_dim=128, conv_taps=4, q_scale=0.125, unit_eps=1e-6,
                                  out_norm_eps=1e-6, decay_rank=16, gate_rank=16, decay_scope="channel", gate="low_rank_sigmoid")
        tensors = {"q": w(64, 128), "k": w(64, 128), "v": w(256, 128), "b": w(2, 128), "o": w(128, 256), "q.conv": w(64, 4) * 8, "k.conv": w(64, 4) * 8,
                   "v.conv": w(256, 4) * 8, "norm": 1 + w(128), "a1": w(16, 128), "a2": w(128, 16) * 4, "g1": w(16, 128), "g2": w(256, 16) * 4,
                   "dt_bias": w(128) * 20 - 4, "A_log": w(2) + 1}
    rt = Runtime(dtype=dtype, device=torch.device("cuda", 0), ops=get_ops())
    part = part_class("mixer", spec)(spec, {n: t.to(dtype) if n not in ("norm", "dt_bias", "A_log") else t for n, t in tensors.items()}, rt)
    return part, torch.randn(400, 128, generator=g).to(dtype).cuda()


def _fed(part, x, cuts, state):
    """The part's outputs for one request whose tokens come in portions that end at `cuts`."""
    out, at = [], 0
    for end in cuts:
        ctx = make_ctx([end - at], [end])
        ctx.prefill_seqs = i32([0] if end - at > 1 else [])
        out.append(part.forward(x[at:end], ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state.view(torch.uint8).view(1, -1), state_slots=i32([0]))))
        at = end
    return torch.cat(out)


@pytest.mark.parametrize("kind", ["plain", "delta"])
def test_float32_recurrences_do_not_depend_on_the_cut(kind):
    part, x = _recurrence_part(kind, torch.float32)
    states = [torch.zeros(part.state_bytes() // 4, device="cuda") for _ in range(2)]
    whole, cut = (_fed(part, x, cuts, s) for cuts, s in zip(([400], [150, 157, 158, 400]), states))
    assert torch.equal(whole, cut) and torch.equal(*states)


@pytest.mark.parametrize("form", ["channel", "head"])
def test_tiles_do_not_depend_on_cuts_at_multiples_of_sixteen(form):
    ops, H, D, V, T = get_ops(), 2, 64, 80, 400
    g = torch.Generator().manual_seed(9)
    y, z = (torch.randn(T, H * (2 * D + V), generator=g) * 0.5).to(torch.bfloat16).cuda(), torch.randn(T, H * D, generator=g).cuda()
    logits = dict(z=None, head_decays=torch.tensor([0.99, 0.8]).cuda()) if form == "head" else dict(head_decays=None)
    results = []
    for cuts in ([T], [176, 208, T]):
        state, out, at = torch.ones(1, H * D * V).cuda(), [], 0
        for end in cuts:
            ctx, binding = _step(state, [end - at])
            ctx.positions += at - int(ctx.positions[0])
            part = y[at:end]
            out.append(ops.linear_recurrence(part[:, :H * D], part[:, H * D:2 * H * D], part[:, 2 * H * D:], ctx, binding, heads=H, dim=D, vdim=V, bias=None,
                                             inv_tau=0.1, q_scale=1.0, k_scale=1.0, **{"z": z[at:end].contiguous(), **logits}))
            at = end
        results.append((torch.cat(out), state))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("kind,entry,tokens", [("plain", "ts_plain_tiles", TILE_TOKENS), ("delta", "ts_channel_tiles", CHANNEL_TILE_TOKENS)])
def test_short_portions_walk_token_by_token(kind, entry, tokens):
    """Two portions and single tokens: either side of the longest portion from which tiles pay."""
    ops = get_ops()
    part, x = _recurrence_part(kind, torch.bfloat16)
    for lens, tiles in (([tokens, 1, 9, 1], True), ([tokens - 1, 1, 9, 1], False)):
        ctx = make_ctx(lens, lens)
        ctx.prefill_seqs = i32([0, 2])
        state = torch.zeros(len(lens), part.state_bytes(), dtype=torch.uint8, device="cuda")
        before = ops.calls.get(entry, 0)
        part.forward(x[:sum(lens)], ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state, state_slots=i32(list(range(len(lens))))))
        assert ops.calls.get(entry, 0) == before + tiles


@pytest.mark.parametrize("bound,tiles", [(256, False), (512, True)])
def test_a_replayed_step_goes_by_its_bound(bound, tiles):
    """Grids of a replayed step are sized by a power of two: what decides whether its portions go by stretches, however long they are."""
    ops = get_ops()
    part, x = _recurrence_part("plain", torch.bfloat16)
    for longest in (60, 256):
        ctx = make_ctx([longest, 1], [longest, 1])
        ctx.prefill_seqs, ctx.replayed, ctx.max_q_len = i32([0, -1]), True, bound
        state = torch.zeros(2, part.state_bytes(), dtype=torch.uint8, device="cuda")
        before = ops.calls.get("ts_plain_tiles", 0)
        part.forward(x[:longest + 1], ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state, state_slots=i32([0, 1])))
        assert ops.calls.get("ts_plain_tiles", 0) == before + tiles


def test_every_tile_of_a_step_has_room_in_the_buffer():
    """The kernels number a request's tiles from cu_q / 16 + its index on; the buffer holds T / 16 + requests + 1."""
    g = torch.Generator().manual_seed(0)
    for _ in range(200):
        lens = torch.randint(0, 50, (int(torch.randint(1, 40, (1,), generator=g)),), generator=g).tolist()
        begin, end = 0, 0
        for s, n in enumerate(lens):
            assert begin // 16 + s >= end
            end = begin // 16 + s + -(-n // 16)
            begin += n
        assert end <= begin // 16 + len(lens) + 1


@pytest.mark.parametrize("kind", ["plain", "delta"])
def test_a_context_that_does_not_say_its_shortest_request(kind):
    part, x = _recurrence_part(kind, torch.bfloat16)
    lens, results = [300, 1], []
    for bare in (False, True):
        ctx = make_ctx(lens, lens)
        ctx.prefill_seqs = i32([0])
        if bare:
            del ctx.min_q_len
        state = torch.zeros(2, part.state_bytes(), dtype=torch.uint8, device="cuda")
        results.append(part.forward(x[:301], ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state, state_slots=i32([0, 1]))))
    assert torch.equal(*results)


@pytest.mark.parametrize("kind", ["plain", "delta"])
def test_beside_tiles_only_single_tokens_are_prepared(kind, monkeypatch):
    """What the walk reads is written for the single tokens of the step and for no others (every new tensor begins as sevens)."""
    part, x = _recurrence_part(kind, torch.bfloat16)
    lens, made, empty = [300, 1, 40, 1], [], torch.empty
    ctx = make_ctx(lens, lens)
    ctx.prefill_seqs = i32([0, 2])
    state = torch.zeros(4, part.state_bytes(), dtype=torch.uint8, device="cuda")

    def sevens(*args, **kwargs):
        t = empty(*args, **kwargs)
        made.append(t.fill_(7) if t.is_floating_point() else t)
        return t

    monkeypatch.setattr(torch, "empty", sevens)
    part.forward(x[:342], ctx, EntryBinding(None, None, 0, 0, 16, 0, state=state, state_slots=i32([0, 1, 2, 3])))
    monkeypatch.undo()
    prepared, = [t for t in made if t.dim() == 3 and t.shape[:2] == (3, 342)]
    written = (prepared != 7).any(dim=2).all(dim=0)
    assert written.nonzero().flatten().tolist() == [300, 341]


def _windowed_latent(heads, dim, rot, rank, window, lens, cached, page, plant=None, sink=False, gate=False, magnitude=1.0):
    """A windowed latent layer over prompt portions: (output, cache rows written, what 64 bits give).  Pages before a window are given back."""
    from tinyserve_llm_b200.config.spec import InlineRotarySpec, LatentAttentionSpec
    from tinyserve_llm_b200.parts.base import Runtime, part_class
    g = torch.Generator().manual_seed(dim + rank + window)
    W, scale, eps = 96, 2.0 / (dim + rot) ** 0.5, 1e-5
    spec = LatentAttentionSpec(hidden_size=W, num_heads=heads, head_dim=dim, rot_dim=rot, value_dim=dim, q_rank=0, kv_rank=rank, scale=scale, window=window,
                               norm_eps=eps, position=InlineRotarySpec(dims=rot), sink=sink, output_gate=gate)
    w = {"q": torch.randn(heads * (dim + rot), W, generator=g) * W ** -0.5, "dkv": torch.randn(rank + rot, W, generator=g) * W ** -0.5,
         "uk": torch.randn(heads * dim, rank, generator=g) * rank ** -0.5, "uv": torch.randn(heads * dim, rank, generator=g) * rank ** -0.5,
         "o": torch.randn(W, heads * dim, generator=g) * (heads * dim) ** -0.5}
    w = {n: t.to(torch.bfloat16) for n, t in w.items()}
    w["dkv.norm"] = 1 + torch.randn(rank, generator=g) * 0.1
    if sink:
        w["sink"] = torch.linspace(-2.0, 6.0, heads)
    if gate:
        w["g"] = (torch.randn(heads * dim, W, generator=g) * W ** -0.5).to(torch.bfloat16)
    rt = Runtime(dtype=torch.bfloat16, device=torch.device("cuda", 0), ops=get_ops())
    part = part_class("mixer", spec)(spec, w, rt)
    part.magnitude = magnitude
    x = torch.randn(sum(lens), W, generator=g).to(torch.bfloat16)
    if plant is not None:
        x[plant, 3] = float("nan")
    ends = [n + c for n, c in zip(lens, cached)]
    counts = [-(-e // page) for e in ends]
    order = torch.randperm(sum(counts) + 1, generator=g).tolist()
    pool = torch.full((sum(counts) + 1, 2, 1, page, rank + rot), float("nan"), dtype=torch.bfloat16)
    history, tables, at = [], [], 0
    for c, n, end in zip(counts, cached, ends):
        ids, at = order[at:at + c], at + c
        rows = torch.randn(n, rank + rot, generator=g).to(torch.bfloat16)
        for j in range(n):
            pool[ids[j // page], 1, 0, j % page] = rows[j]
        history.append(rows)
        gone = max(0, n - window + 1) // page
        for i in ids[:gone]:
            pool[i] = float("nan")
        tables.append([-1] * gone + ids[gone:] + [-1] * (max(counts) - c))
    ctx = make_ctx(lens, ends)
    ctx.replayed, ctx.prefill_seqs = False, i32([s for s, n in enumerate(lens) if n > 1])
    per = page * (rank + rot)
    dev = pool.cuda()
    binding = EntryBinding(dev, None, 2 * per, per, page, pool.shape[0], i32(tables), max(counts))
    before = rt.ops.calls.get("ts_prefill_attention_tcgen05_dense", 0)
    got = part.forward(x.cuda(), ctx, binding)
    assert rt.ops.calls.get("ts_prefill_attention_tcgen05_dense", 0) == before + 1
    if plant is not None:
        return got.cpu(), None
    d = {n: t.double() for n, t in w.items()}
    freq = 10000.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)

    def turned(t, positions):                            # [n, k, rot]
        a = positions.double()[:, None, None] * freq
        u, v = t.chunk(2, dim=-1)
        return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1) * magnitude

    want, at = [], 0
    for n, c, rows in zip(lens, cached, history):
        xs, positions = x[at:at + n].double(), torch.arange(c, c + n)
        q, y = (xs @ d["q"].t()).view(n, heads, dim + rot), xs @ d["dkv"].t()
        lat = y[:, :rank] / (y[:, :rank].pow(2).mean(-1, keepdim=True) + eps).sqrt() * d["dkv.norm"]
        new = torch.cat([lat, turned(y[:, None, rank:], positions)[:, 0]], dim=-1)
        full = torch.cat([rows.double(), new])
        k = torch.cat([(full[:, :rank] @ d["uk"].t()).view(-1, heads, dim), full[:, None, rank:].expand(-1, heads, -1)], dim=-1)
        q = torch.cat([q[..., :dim], turned(q[..., dim:], positions)], dim=-1)
        s = torch.einsum("ihd,jhd->hij", q, k) * scale
        j = torch.arange(c + n)[None]
        s = s.masked_fill((j > positions[:, None]) | (j <= positions[:, None] - window), -float("inf"))
        if sink:                                         # a score without a key or a value
            s = torch.cat([s, d["sink"][:, None, None].expand(-1, n, 1)], dim=-1)
        o = torch.einsum("hij,jhd->ihd", torch.softmax(s, -1)[..., :c + n], (full[:, :rank] @ d["uv"].t()).view(-1, heads, dim)).reshape(n, -1)
        want.append((o * torch.sigmoid(xs @ d["g"].t()) if gate else o) @ d["o"].t())
        at += n
    return got.double().cpu(), torch.cat(want)


@pytest.mark.parametrize("heads,dim,rot,rank,window,lens,cached,page", [
    (2, 128, 64, 512, 100, [300, 1, 129, 2], [0, 500, 777, 130], 64), (3, 64, 24, 40, 1, [140], [260], 16), (1, 128, 40, 72, 1000, [150, 150], [0, 1300], 256),
    (2, 64, 16, 64, 129, [128, 257], [127, 1], 64), (4, 128, 8, 128, 4096, [513], [64], 128)])
def test_windowed_latent_portions_on_keys_and_values_of_their_own(heads, dim, rot, rank, window, lens, cached, page):
    """Windows inside a key tile, over several, wider than the context; portions behind cached keys whose early pages are given back."""
    got, want = _windowed_latent(heads, dim, rot, rank, window, lens, cached, page)
    # bfloat16 queries, latents, keys, values, weights, heads and outputs: seven roundings of at most 2^-9, half of that on average; in a
    # single row scores of up to 8 (two is their deviation), off by up to 2^-9 of themselves, move its weights by as much as 8 2^-9 more
    err, off = (got - want).norm(dim=-1) / want.norm(dim=-1), float((got - want).norm() / want.norm())
    assert float(err.max()) < 15 * 2.0 ** -9 and off < 3.5 * 2.0 ** -9, (float(err.max()), off)


@pytest.mark.parametrize("heads,dim", [(3, 128), (2, 64)])
@pytest.mark.parametrize("options", [{"sink": True}, {"gate": True}, {"magnitude": 1.4}, {"sink": True, "gate": True, "magnitude": 0.8}])
def test_windowed_latent_portions_with_sinks_gates_and_magnitudes(heads, dim, options):
    """The options of the layers without a window.  Bounds as above; sinks and gates make outputs smaller and round once more."""
    got, want = _windowed_latent(heads, dim, 32, 128, 90, [200, 1, 150], [0, 70, 333], 64, **options)
    err, off = (got - want).norm(dim=-1) / want.norm(dim=-1), float((got - want).norm() / want.norm())
    assert float(err.max()) < 15 * 2.0 ** -9 and off < 4 * 2.0 ** -9, (float(err.max()), off)


def test_a_latent_that_is_not_finite_reaches_the_queries_that_see_it_only():
    sizes = (2, 128, 64, 256, 70, [400, 130], [30, 0], 64)
    (clean, _), (got, _) = _windowed_latent(*sizes), _windowed_latent(*sizes, plant=201)
    sees = torch.zeros(530, dtype=torch.bool)
    sees[201:271] = True
    assert torch.isnan(got[sees]).all() and torch.equal(got[~sees], clean[~sees].to(got.dtype))


def _both_forms(heads, dim, rot, rank, window, lens, cached, deviation):
    """Relative errors against 64 bits of windowed latent attention alone, its scores of this deviation: (unfolded, folded), each (worst row, all)."""
    from tinyserve_llm_b200.config.spec import InlineRotarySpec, LatentAttentionSpec
    from tinyserve_llm_b200.parts.base import Runtime, part_class
    g, page, T = torch.Generator().manual_seed(rank + dim), 64, sum(lens)
    normal = lambda *shape, std=1.0: (torch.randn(shape, generator=g) * std).to(torch.bfloat16)
    spec = LatentAttentionSpec(hidden_size=64, num_heads=heads, head_dim=dim, rot_dim=rot, value_dim=dim, q_rank=0, kv_rank=rank,
                               scale=deviation / (dim + rot) ** 0.5, window=window, norm_eps=1e-5, position=InlineRotarySpec(dims=rot))
    w = {"q": normal(heads * (dim + rot), 64), "dkv": normal(rank + rot, 64), "uk": normal(heads * dim, rank, std=rank ** -0.5),
         "uv": normal(heads * dim, rank, std=rank ** -0.5), "o": normal(64, heads * dim), "dkv.norm": torch.ones(rank)}
    part = part_class("mixer", spec)(spec, w, Runtime(dtype=torch.bfloat16, device=torch.device("cuda", 0), ops=get_ops()))
    ends = [n + c for n, c in zip(lens, cached)]
    counts = [-(-e // page) for e in ends]
    pool, q = normal(sum(counts), 1, 1, page, rank + rot), normal(T, heads * (dim + rot))
    tables = [list(range(sum(counts[:s]), sum(counts[:s + 1]))) + [-1] * (max(counts) - n) for s, n in enumerate(counts)]
    binding = EntryBinding(pool.cuda(), None, page * (rank + rot), 0, page, pool.shape[0], i32(tables), max(counts))
    freq = 10000.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
    want, at = [], 0
    for s, (n, c) in enumerate(zip(lens, cached)):
        full = pool.view(-1, page, rank + rot)[tables[s][:counts[s]]].reshape(-1, rank + rot)[:c + n].double()
        positions = torch.arange(c, c + n)
        turned = q[at:at + n].double().view(n, heads, dim + rot)
        a, (u, v) = positions.double()[:, None, None] * freq, turned[..., dim:].chunk(2, dim=-1)
        turned = torch.cat([turned[..., :dim], u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)
        k = torch.cat([(full[:, :rank] @ w["uk"].double().t()).view(-1, heads, dim), full[:, None, rank:].expand(-1, heads, -1)], dim=-1)
        j = torch.arange(c + n)[None]
        scores = torch.einsum("ihd,jhd->hij", turned, k) * spec.scale
        scores = scores.masked_fill((j > positions[:, None]) | (j <= positions[:, None] - window), -float("inf"))
        want.append(torch.einsum("hij,jhd->ihd", torch.softmax(scores, -1), (full[:, :rank] @ w["uv"].double().t()).view(-1, heads, dim)))
        at += n
    want, results = torch.cat(want), []
    for replayed in (False, True):                       # a step that is replayed stays on the folded form
        ctx = make_ctx(lens, ends)
        ctx.replayed, ctx.prefill_seqs = replayed, i32([s for s, n in enumerate(lens) if n > 1])
        before = get_ops().calls.get("ts_prefill_attention_tcgen05_dense", 0)
        got = part.attend(q.cuda(), ctx, binding).double().cpu().view(T, heads, dim)
        assert get_ops().calls.get("ts_prefill_attention_tcgen05_dense", 0) == before + (not replayed)
        off = (got - want).norm(dim=-1) / want.norm(dim=-1)
        results.append((float(off.max()), float((got - want).norm() / want.norm())))
    return results


@pytest.mark.parametrize("deviation", [1.0, 3.0, 6.0])
@pytest.mark.parametrize("heads,dim,rot,rank,window,lens,cached", [(4, 128, 64, 512, 256, [512], [0]), (3, 64, 32, 256, 100, [200, 150], [333, 0])])
def test_keys_worked_out_for_a_step_are_no_further_from_64_bits_than_the_latents(heads, dim, rot, rank, window, lens, cached, deviation):
    """
    Flat and peaked scores.  Both forms round the outputs once to bfloat16 and, before that, the values or their weighted sum; with nothing
    else rounded to less than two such pieces they differ by the luck of those roundings, hundredths over 10^5 of them.
    """
    (worst, off), (folded_worst, folded) = _both_forms(heads, dim, rot, rank, window, lens, cached, deviation)
    assert off <= 1.02 * folded and worst <= 1.5 * folded_worst, (off, folded, worst, folded_worst)


@pytest.mark.parametrize("rows,rank,cols,low", [(1, 40, 8, 8), (129, 72, 256, 128), (300, 512, 1032, 0), (2048, 512, 4096, 2048), (2900, 128, 10240, 5120)])
def test_products_in_pieces(rows, rank, cols, low):
    """Every tile shape of the product (one tile of rows, narrow, wide, pairs of CTAs), pieces of all, half and none of its columns."""
    g = torch.Generator().manual_seed(rows)
    x, w = torch.randn(rows, rank, generator=g).to(torch.bfloat16), (torch.randn(cols, rank, generator=g) * rank ** -0.5).to(torch.bfloat16)
    y = get_ops().gemm_tcgen05_pieces(x.cuda(), w.cuda(), low)
    want = (x.double().cuda() @ w.double().cuda().t())
    # float32 sums of `rank` terms of about rank^-1/2: within sqrt(rank) 2^-24 of one; the sum of two pieces within 2^-17 of itself, a single one 2^-9
    sums = rank ** 0.5 * 2.0 ** -22
    assert bool(((y[:, :cols].double() - want).abs() <= want.abs() * 2.0 ** -8 + sums).all())
    both = y[:, :low].double() + y[:, cols:].double()
    assert bool(((both - want[:, :low]).abs() <= want[:, :low].abs() * 2.0 ** -16 + sums).all())


def _latent_part(heads, dim, rot, rank, window, **extra):
    from tinyserve_llm_b200.config.spec import InlineRotarySpec, LatentAttentionSpec
    from tinyserve_llm_b200.parts.base import Runtime, part_class
    g, gate = torch.Generator().manual_seed(heads + rank), extra.get("output_gate", False)
    w = lambda *shape: (torch.randn(shape, generator=g) * shape[-1] ** -0.5).to(torch.bfloat16)
    tensors = {"q": w(heads * (dim + rot), 96), "dkv": w(rank + rot, 96), "uk": w(heads * dim, rank), "uv": w(heads * dim, rank), "o": w(96, heads * dim),
               "dkv.norm": torch.ones(rank)}
    if gate:
        tensors["g"] = w(heads * dim, 96)
    spec = LatentAttentionSpec(hidden_size=96, num_heads=heads, head_dim=dim, rot_dim=rot, value_dim=dim, q_rank=0, kv_rank=rank,
                               scale=(dim + rot) ** -0.5, window=window, norm_eps=1e-5, position=InlineRotarySpec(dims=rot), **extra)
    return part_class("mixer", spec)(spec, tensors, Runtime(dtype=torch.bfloat16, device=torch.device("cuda", 0), ops=get_ops()))


def test_a_windowed_portion_takes_its_form_whatever_else_is_in_the_step():
    """A portion's own tokens and keys decide, and a portion that a replayed step may hold stays with the form of such steps."""
    part = _latent_part(2, 128, 64, 128, 300)
    for tokens, cached, limit, unfolded in ((128, 0, 0, True), (127, 0, 0, False), (128, 90000, 0, True), (512, 0, 512, False), (513, 0, 512, True),
                                            (700, 5000, 512, True), (700, 5000, 1024, False)):
        for lens, kept in (([], []), ([600], [0]), ([2, 1, 40], [0, 9, 3000]), ([1] * 9, [5] * 9), ([2000, 64], [0, 70000])):
            lens, kept = [tokens] + lens, [cached] + kept
            ctx = make_ctx(lens, [n + c for n, c in zip(lens, kept)])
            ctx.replayed, ctx.replay_limit = False, limit
            q = torch.empty(sum(lens), 2 * 192, dtype=torch.bfloat16, device="cuda")
            assert (0 in part.unfolded_requests(q, ctx)) == unfolded, (tokens, cached, limit, lens)
    far = _latent_part(2, 128, 64, 128, 20000)           # a window of 20,000 keys for 200 tokens: the latents are read as they are
    ctx = make_ctx([200, 2000], [50000, 2000])
    ctx.replayed = False
    assert far.unfolded_requests(torch.empty(2200, 2 * 192, dtype=torch.bfloat16, device="cuda"), ctx) == [1]


def test_the_engine_says_which_steps_it_may_replay():
    from types import SimpleNamespace
    from tinyserve_llm_b200.engine.step import HostView, StepContext
    host = HostView([0], [0, 3], [0], [3], [0])
    for runner, limit in ((None, 0), (SimpleNamespace(cuda_graphs=True, graph_max_tokens=512), 512), (SimpleNamespace(cuda_graphs=False, graph_max_tokens=512), 0)):
        assert StepContext(runner, 3, 1, host).replay_limit == limit


@pytest.mark.parametrize("rank", [512, 128])             # folded portions four tokens a CTA, and a token a CTA
def test_portions_of_both_forms_in_one_step(rank):
    """Long portions beside short ones and single tokens: every row as in a step in which its request is alone with its like."""
    part, lens, cached, page = _latent_part(2, 128, 64, rank, 200), [700, 300, 1, 90, 600], [0, 40, 333, 10, 77], 64
    g = torch.Generator().manual_seed(rank)
    ends = [n + c for n, c in zip(lens, cached)]
    counts = [-(-e // page) for e in ends]
    pool = torch.randn(sum(counts), 1, 1, page, rank + 64, generator=g).to(torch.bfloat16).cuda()
    q = torch.randn(sum(lens), 2 * 192, generator=g).to(torch.bfloat16).cuda()
    tables = [list(range(sum(counts[:s]), sum(counts[:s + 1]))) + [-1] * (max(counts) - n) for s, n in enumerate(counts)]

    def attend(which):
        ctx = make_ctx([lens[s] for s in which], [ends[s] for s in which])
        ctx.replayed, ctx.replay_limit, ctx.prefill_seqs = False, 512, i32([i for i, s in enumerate(which) if lens[s] > 1])
        rows = torch.cat([torch.arange(sum(lens[:s]), sum(lens[:s + 1])) for s in which]).cuda()
        out = part.attend(q[rows].contiguous(), ctx, EntryBinding(pool, None, page * (rank + 64), 0, page, pool.shape[0], i32([tables[s] for s in which]), max(counts)))
        return out, torch.split(out, [lens[s] for s in which])

    before = dict(get_ops().calls)
    together, rows = attend([0, 1, 2, 3, 4])
    assert torch.isfinite(together).all()
    for name in ("ts_prefill_attention_tcgen05_dense", "ts_latent_attention"):
        assert get_ops().calls[name] == before.get(name, 0) + 1
    _, (first, last) = attend([0, 4])
    assert torch.equal(rows[0], first) and torch.equal(rows[4], last)
    # the folded form's products of other numbers of rows may sum in another order, in float32, before one rounding to bfloat16
    _, others = attend([1, 2, 3])
    for got, want in zip((rows[1], rows[2], rows[3]), others):
        assert float((got.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -9


def test_queries_of_unfolded_portions_are_rotated_by_their_positions():
    """A context's positions, which need not be the tokens' places among the keys."""
    part, lens, page = _latent_part(2, 64, 24, 128, 100), [130, 1, 200], 64
    ctx = make_ctx(lens, [150, 9, 200])
    ctx.replayed, ctx.prefill_seqs = False, i32([0, 2])
    ctx.positions += 1000
    pool = torch.zeros(8, 1, 1, page, 152, dtype=torch.bfloat16, device="cuda")
    binding = EntryBinding(pool, None, page * 152, 0, page, 8, i32([[0, 1, 2, -1], [3, -1, -1, -1], [4, 5, 6, 7]]), 4)
    _, (turn, _), _, _ = get_ops().latent_gather(ctx, binding, 350, 200, 128, 24, 100, part.frequencies, 0.75)
    angles = ctx.positions.double()[:, None] * part.frequencies.double()
    for s, (a, b) in enumerate(((0, 130), (131, 331))):
        want = 0.75 * torch.stack([angles[a:b].cos(), angles[a:b].sin()], dim=-1)
        # an angle of up to 1,200 is a float32 product, within 2^-14 of itself; cosine and sine follow it
        assert float((turn[a:b, :12].double() - want).abs().max()) < 2.0 ** -13


@pytest.mark.parametrize("kind", ["delta", "channel"])
def test_a_delta_walk_whose_wait_runs_out_stores_nothing(kind):
    """A limit of no time at all: every CTA gives up at its first tile, waits for its copies, and leaves the state as it was."""
    ops, H, D, lens = get_ops(), 2, 64, [40, 17, 1, 2]
    g = torch.Generator().manual_seed(1)
    T = sum(lens)
    y, z, b, gates = (torch.randn(T, n, generator=g).cuda() for n in (3 * H * D, H * D, H, 2 * H))
    per_head, per_channel = torch.zeros(H).cuda(), torch.zeros(H * D).cuda()
    state = torch.randn(len(lens) + 3, H * D * D, generator=g).cuda()
    sizes = dict(heads=H, kv_heads=H, dim=D, vdim=D, unit_eps=1e-6, q_scale=0.25)
    parts, held, results = y.split(H * D, dim=1), state.clone(), []
    for limit in ({"wait_cycles": 0}, {}, {}):
        ctx, binding = _step(held, lens)
        if kind == "delta":
            results.append(ops.delta_tiles(*parts, gates, per_head, per_head, ctx, binding, **sizes, **limit))
        else:
            results.append(ops.channel_tiles(*parts, z, b, per_channel, per_head, ctx, binding, **sizes, **limit))
        torch.cuda.synchronize()
        if limit:
            assert torch.equal(held, state)
            with pytest.raises(KernelError, match="delta_tiles"):
                ops.check_device_errors()
        else:
            assert not torch.equal(held, state)
            ops.check_device_errors()
            held = state.clone()
    rows = [t for s, n in enumerate(lens) for t in range(sum(lens[:s]), sum(lens[:s + 1])) if n > 1]
    assert torch.equal(results[1][rows], results[2][rows])
