"""
Attention over a cached latent: per token the cache keeps c = norm(W_dkv h)[:kv_rank] and one rotated
key part k_rot shared by all heads; a head's keys and values are W_uk,h c and W_uv,h c.

    c_q = norm(W_dq h),  q = W_uq c_q  laid out per head as [head_dim unrotated | rot_dim rotated]
    score_h(i, j) = (q_flat,h(i) . W_uk,h c(j) + rot(q_rot,h(i)) . k_rot(j)) * scale
    y = W_o concat_h( W_uv,h sum_j softmax_j(score_h(i, .)) c(j) )

Since q_flat . (W_uk c) = (W_uk^T q_flat) . c, the engine folds W_uk into the query (one batched
product per step) and W_uv into the output of the attention (another), and the attention kernel
works on cache rows [c | k_rot] directly: keys and values of a head are never materialised, in prompts
as in decoding.  The cache entry is one "kv head" of kv_rank + rot_dim channels without a value pool;
a window makes it a layer group of its own whose pages are given back as the window passes.

Options of the description: `q_rank` 0 makes the queries a projection of the input, q = W_q h, without a
latent and a norm of their own; `rot_dim` 0 leaves out the rotated part (attention without positions: the
cache row is c alone and no position part is built); `output_gate` multiplies the concatenated heads by
sigmoid(W_g h), read from the same input as the other projections, before W_o; `sink` adds exp(sink_h) to every
softmax's sum of head h.  A rotation of neighbouring channels is a rotation by halves of channels put in another
order: the rows of W_dkv and W_q that make the rotated parts are reordered when the part is built (a score is a sum
over the channels, so the order does not show), and the kernels rotate by halves throughout.

Prompt portions of a step that is launched once (not replayed from a CUDA graph) take another way where the
sizes allow (bfloat16, key and value heads of one size the tcgen05 prompt kernel takes, up to 64 rotated channels): the
latents the portions see, their whole contexts or what a window leaves, are gathered from the pages (their rotated parts, one for
all heads, go to the kernel as they lie), a head's keys and values are worked out for the step ([K | V] = C [W_uk; W_uv]^T, one
product, behind a window with keys of two pieces: a quarter of the folded form's arithmetic at a latent of 512 channels and heads of 128) and the tcgen05 prompt kernel
attends over them; requests that feed one token in the same step stay on the folded form, and so do, behind a window, portions that a
replayed step may hold or that see many keys for their tokens.  The two ways differ by rounding only.

Tensors (local names): dq, dq.norm, uq (or q), dkv, dkv.norm, uk, uv, o, g with an output gate, sink.
"""

from __future__ import annotations

import copy

import torch

from tinyserve_llm_b200.config.spec import LatentAttentionSpec
from tinyserve_llm_b200.parts.base import KVNeed, Mixer, Runtime, TensorDecl, part_class, register_part
from tinyserve_llm_b200.parts.linear import Linear, fuse_rows

MAX_KV_RANK = 512       # csrc/attention_latent.cu: 16 output channels a lane
MATERIALIZE_MIN_TOKENS = 128    # prompt portions of a step, together (with a window: each), from which keys and values are worked out for the step
# With a window: keys a token a portion feeds, up to which they are.  The attention alone, heads of 128, latent of 512, us folded / unfolded, 8 heads
# and 16: 128 tokens, 9 keys a token 115 / 71, 123 / 72; 33 keys 349 / 150, 410 / 170; 513 tokens, 9 keys 688 / 153, 693 / 172; 2,048 tokens, 3 keys
# 2,693 / 164, 2,728 / 327.  Beyond that the latents gathered for few tokens cost more than they save (three portions of 160 .. 290 tokens, windows
# of 1,024: 163 / 336 at 95 keys a token fed).
MATERIALIZE_MAX_KEYS = 32


def evens_then_odds(rows: torch.Tensor) -> torch.Tensor:
    """[..., 2n, columns] with rows 0, 2, 4, ... first, then 1, 3, 5, ...: neighbours become halves."""
    return torch.cat([rows[..., 0::2, :], rows[..., 1::2, :]], dim=-2)


@register_part("mixer", "latent_attention")
class LatentAttention(Mixer):
    graph_safe = True

    @classmethod
    def validate(cls, spec: LatentAttentionSpec) -> None:
        if spec.kv_rank > MAX_KV_RANK:
            raise ValueError(f"kv_rank={spec.kv_rank} is not supported: the latent attention kernel takes up to {MAX_KV_RANK}")
        if spec.rot_dim % 2 or spec.rot_dim < 0 or spec.q_rank < 0:
            raise ValueError(f"rot_dim={spec.rot_dim} must be even and q_rank={spec.q_rank} not negative")
        if (spec.rot_dim > 0) != (spec.position is not None):
            raise ValueError("latent attention: a rotated key part and a position part come together")

    @classmethod
    def declare(cls, spec: LatentAttentionSpec) -> dict[str, TensorDecl]:
        cls.validate(spec)
        H, D, R, V = spec.num_heads, spec.head_dim, spec.rot_dim, spec.value_dim
        out = {
            "dkv": TensorDecl((spec.kv_rank + R, spec.hidden_size)), "dkv.norm": TensorDecl((spec.kv_rank,), init="unit"),
            "uk": TensorDecl((H * D, spec.kv_rank)), "uv": TensorDecl((H * V, spec.kv_rank)),
            "o": TensorDecl((spec.hidden_size, H * V)),
        }
        if spec.q_rank > 0:
            out.update({"dq": TensorDecl((spec.q_rank, spec.hidden_size)), "dq.norm": TensorDecl((spec.q_rank,), init="unit"),
                        "uq": TensorDecl((H * (D + R), spec.q_rank))})
        else:
            out["q"] = TensorDecl((H * (D + R), spec.hidden_size))
        if spec.output_gate:
            out["g"] = TensorDecl((H * V, spec.hidden_size))
        if spec.sink:
            out["sink"] = TensorDecl((H,))
        return out

    def __init__(self, spec: LatentAttentionSpec, tensors: dict[str, torch.Tensor], rt: Runtime) -> None:
        super().__init__(spec, tensors, rt)
        self.validate(spec)
        H, D, V, rank = spec.num_heads, spec.head_dim, spec.value_dim, spec.kv_rank
        R = spec.rot_dim
        self.position = None
        if spec.position is not None:
            self.position = part_class("position", spec.position)(spec.position, {}, rt)
            if getattr(self.position, "frequencies", None) is None or self.position.dims != R:
                raise NotImplementedError("latent attention rotates inside its kernels: it takes a position part with "
                                          "`frequencies` over exactly rot_dim channels")
        self.frequencies = getattr(self.position, "frequencies", None)
        self.magnitude = float(getattr(self.position, "magnitude", 1.0))
        q_name = "uq" if spec.q_rank > 0 else "q"
        q_rows, dkv_rows = tensors[q_name], tensors["dkv"]
        if getattr(self.position, "interleaved", False):
            by_head = q_rows.view(H, D + R, -1)
            q_rows = torch.cat([by_head[:, :D], evens_then_odds(by_head[:, D:])], dim=1).reshape(q_rows.shape)
            dkv_rows = torch.cat([dkv_rows[:rank], evens_then_odds(dkv_rows[rank:])], dim=0)
        # one product of the input: columns [c_q raw (or q) | c raw | k_rot raw | gate logits]
        rows = [tensors["dq"] if spec.q_rank > 0 else q_rows, dkv_rows] + ([tensors["g"]] if spec.output_gate else [])
        self.down = Linear(fuse_rows(rows), rt)
        self.q_norm = self.up_q = None
        if spec.q_rank > 0:
            self.q_norm = tensors["dq.norm"].to(device=rt.device, dtype=torch.float32).contiguous()
            self.up_q = Linear(q_rows, rt)
        self.kv_norm = tensors["dkv.norm"].to(device=rt.device, dtype=torch.float32).contiguous()
        # W_uk per head, transposed to [H, rank, D]: the product that folds it into the query reads rows of D
        self.uk_t = tensors["uk"].to(device=rt.device, dtype=rt.dtype).view(H, D, rank).transpose(1, 2).contiguous()
        # the unfolded form of prompt portions: [W_uk; W_uv] as stored, one product for keys and values (its second half is self.uv's
        # memory); rotated parts go to the kernel as TMA sub-tiles of 64 channels: rows on 16-byte boundaries
        self.uk_uv = None
        if D == V and R <= 64 and R % 8 == 0 and (R == 0 or rank % 8 == 0):
            self.uk_uv = torch.cat([tensors[n].to(device=rt.device, dtype=rt.dtype).reshape(H * D, rank) for n in ("uk", "uv")])
            self.uv = self.uk_uv[H * D:].view(H, V, rank)
        else:
            self.uv = tensors["uv"].to(device=rt.device, dtype=rt.dtype).view(H, V, rank).contiguous()
        self.out = Linear(tensors["o"], rt)
        self.sink = tensors["sink"].to(device=rt.device, dtype=torch.float32).contiguous() if spec.sink else None

    def kv_need(self) -> KVNeed:
        return KVNeed(1, self.spec.kv_rank + self.spec.rot_dim, self.spec.window, values=False)

    # ------------------------------------------------------------------ prompt portions on keys and values of their own
    def unfolded_requests(self, q: torch.Tensor, ctx) -> list[int]:
        """
        The requests whose prompt portions attend over keys and values worked out for the step.  With a window that follows from the portion
        alone, its tokens and the keys the window leaves it, so that a row's form does not depend on what else is in the step: a portion
        that a step replayed from a graph may hold stays on the folded form, which such a step takes, in every step.
        """
        spec, host, ops = self.spec, getattr(ctx, "host", None), self.rt.ops
        # (small steps leave first: they are bound by the host)
        if (host is None or host.cu_q[-1] < MATERIALIZE_MIN_TOKENS or getattr(ctx, "replayed", True) or ctx.max_q_len <= 1
                or self.uk_uv is None or (spec.window and not spec.rot_dim)
                or not ops.dense_prompt_attention_supported(q, spec.num_heads, spec.num_heads, spec.head_dim)):
            return []
        # (windows come in the kernel's form with a rotated part, whose queries, keys and probabilities have the folded form's precision)
        lens = [b - a for a, b in zip(host.cu_q, host.cu_q[1:])]
        portions = [s for s, n in enumerate(lens) if n > 1]
        if not spec.window:
            return portions if sum(lens[s] for s in portions) >= MATERIALIZE_MIN_TOKENS else []
        least = max(MATERIALIZE_MIN_TOKENS, getattr(ctx, "replay_limit", 0) + 1)
        return [s for s in portions if lens[s] >= least and self._keys_of(host, s) <= MATERIALIZE_MAX_KEYS * lens[s]]

    def _keys_of(self, host, s: int) -> int:
        """How many keys of a request are gathered for its portion."""
        return host.ctx_lens[s] - self.rt.ops.latent_first_key(host.ctx_lens[s], host.cu_q[s + 1] - host.cu_q[s], self.spec.window)

    @staticmethod
    def _divided(ctx, unfolded: list[int]):
        """The step's context for the folded form, tokens of the unfolded requests marked as padding rows (that form skips them), and for the unfolded one."""
        host = ctx.host
        lens = [b - a for a, b in zip(host.cu_q, host.cu_q[1:])]
        rest = [n for s, n in enumerate(lens) if s not in set(unfolded)]
        flags = torch.zeros(len(lens), dtype=torch.bool)
        flags[unfolded] = True
        flags = flags.pin_memory().to(ctx.cu_q.device, non_blocking=True)
        of_token = flags[ctx.seq_of_token.long().clamp_min(0)]
        folded, others = copy.copy(ctx), copy.copy(ctx)
        folded.seq_of_token = torch.where(of_token, -1, ctx.seq_of_token)
        folded.min_q_len, folded.max_q_len = min(rest), max(rest)
        listed = getattr(ctx, "prefill_seqs", None)
        if any(n > 1 for n in rest):                     # portions on both forms
            listed = torch.arange(len(lens), dtype=torch.int32, device=ctx.cu_q.device) if listed is None else listed
            others.prefill_seqs = torch.where(flags[listed.long().clamp_min(0)], listed, -1)
        return folded, others

    def _attend_unfolded(self, q: torch.Tensor, ctx, binding, unfolded: list[int], out: torch.Tensor | None) -> torch.Tensor:
        spec, ops = self.spec, self.rt.ops
        H, D, R, rank = spec.num_heads, spec.head_dim, spec.rot_dim, spec.kv_rank
        keys = [self._keys_of(ctx.host, s) for s in unfolded]
        c, shared, odd, kv_start = ops.latent_gather(ctx, binding, sum(keys), max(keys), rank, R, spec.window, self.frequencies, self.magnitude)
        if not spec.window:
            kv, k_low = ops.linear(c, self.uk_uv), None     # [keys, H D | H D]
        else:                                               # keys as two pieces: the folded form rounds none
            kv = ops.gemm_tcgen05_pieces(c, self.uk_uv, H * D)
            k_low = kv[:, 2 * H * D:]
        return ops.dense_prompt_attention(q, kv[:, :H * D], kv[:, H * D:2 * H * D], kv_start, ctx, H, H, D, spec.scale, out, q_head_cols=D + R,
                                          shared=shared, sink=self.sink, window=spec.window, odd_rows=odd, k_low=k_low)

    def attend(self, q: torch.Tensor, ctx, binding) -> torch.Tensor:
        """[T, H V] in q's dtype: the heads' outputs for queries q [T, H (D + R)], rotated here, over the cached rows [c | k_rot]."""
        spec, ops = self.spec, self.rt.ops
        H, D, R, V, rank = spec.num_heads, spec.head_dim, spec.rot_dim, spec.value_dim, spec.kv_rank
        unfolded = self.unfolded_requests(q, ctx)
        if unfolded and len(unfolded) == len(ctx.host.ctx_lens):
            return self._attend_unfolded(q, ctx, binding, unfolded, None)
        folded_ctx, unfolded_ctx = self._divided(ctx, unfolded) if unfolded else (ctx, None)
        q_lat = ops.per_head_linear(q, self.uk_t, H, D + R, D)            # float32 [T, H, rank]: W_uk^T q_flat
        o_lat = ops.latent_attention(q_lat, q, folded_ctx, binding, H, D + R, D, rank, R, self.frequencies, spec.scale,
                                     spec.window, magnitude=self.magnitude, sink=self.sink)   # [T, H, rank]: softmax-weighted sums of c
        o = ops.per_head_linear(o_lat.view(-1, H * rank), self.uv, H, rank, rank, out_dtype=q.dtype)   # [T, H, V]
        o = o.reshape(-1, H * V)
        if not unfolded:
            return o
        return self._attend_unfolded(q, unfolded_ctx, binding, unfolded, o.contiguous())      # those portions' rows are written over

    def forward(self, x: torch.Tensor, ctx, binding) -> torch.Tensor:
        spec, ops = self.spec, self.rt.ops
        H, D, R, V, rank = spec.num_heads, spec.head_dim, spec.rot_dim, spec.value_dim, spec.kv_rank
        y = self.down(x)                                                  # [T, (q_rank or H (D + R)) + rank + R (+ H V)]
        if spec.q_rank > 0:
            latents = spec.q_rank + rank + R
            c_q = ops.latent_prepare(y[:, :latents], ctx, binding, spec.q_rank, rank, R, self.q_norm, self.kv_norm,
                                     spec.norm_eps, self.frequencies, self.magnitude)   # normed query latent; [c | k_rot] is in the cache
            q = self.up_q(c_q)                                            # [T, H (D + R)]
        else:
            latents = H * (D + R) + rank + R
            q = y[:, :H * (D + R)]
            ops.latent_prepare(y[:, H * (D + R):latents], ctx, binding, 0, rank, R, None, self.kv_norm, spec.norm_eps,
                               self.frequencies, self.magnitude)
        o = self.attend(q, ctx, binding)
        if spec.output_gate:
            o = ops.sigmoid_gate(o, y[:, latents:latents + H * V])
        return self.out(o)
