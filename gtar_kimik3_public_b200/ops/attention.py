"""Attention over the paged cache: picks the kernel for the step's shape and dtype.

* float32, or a head size the tensor-core kernels do not take: the exact kernel (any cut of the
  work gives bit-equal results);
* bfloat16, every sequence bringing one token: the split-KV decode kernel;
* bfloat16 otherwise (prompts, or continuations of several tokens): the flash prefill kernel.

Layers that keep one latent row per position for all heads (``latent_attention`` below): bfloat16 rows whose sizes the
tensor-core kernel takes go there, prompts and single tokens alike (single-token steps cut into splits); everything else, and
every float32 run, goes to the exact latent kernel.
"""

from __future__ import annotations

import os

import torch

from . import functional as F

FAST_HEAD_DIMS = (64, 128)


def fused_decode_ok(qkv: torch.Tensor, kv: F.PagedKV, n_q: int, n_kv: int, head_dim: int) -> bool:
    """Whether the decode kernel that also norms, rotates and writes the new token can take the layer."""
    return (qkv.dtype == torch.bfloat16 and kv.k.dtype == torch.bfloat16 and head_dim in FAST_HEAD_DIMS
            and kv.page_size == 64 and n_q // n_kv <= 16)


def decode_split_count(ctx, n_kv: int, kv: F.PagedKV) -> int:
    """Blocks that share a sequence's pages in this layer: from the layer's own kv heads and the step's sequence
    lengths (in a captured step the middle of the lengths that the shape's bound covers, not the lengths of the
    day)."""
    sms = F.sm_count(kv.k.device)
    length = ctx.typical_kv_len or ctx.max_kv_len
    return F.decode_splits(ctx.n_seqs, n_kv, length, kv.page_size, sms, F.decode_cluster_places(kv.k.shape[3], sms))


# "auto": the evenly dealt kernel where the estimate favours it; "always" / "never" for measurements
DECODE_FLAT = os.environ.get("GTAR_B200_DECODE_FLAT", "auto")


def decode_flat_preferred(ctx, n_kv: int, kv: F.PagedKV) -> bool:
    """Whether the step's decode attention deals the pages of all sequences out evenly (one kernel, partial
    results through scratch) instead of giving every (sequence, kv head) pair the same number of blocks."""
    if DECODE_FLAT != "auto":
        return DECODE_FLAT == "always"
    sms = F.sm_count(kv.k.device)
    length = ctx.typical_kv_len or ctx.max_kv_len
    return F.decode_flat_wins(ctx.n_seqs, n_kv, length, kv.page_size, sms, F.decode_cluster_places(kv.k.shape[3], sms),
                              F.decode_flat_places(kv.k.shape[3], sms))


def paged_attention(q: torch.Tensor, kv: F.PagedKV, ctx, scale: float, window: int = 0, sink: bool = False) -> torch.Tensor:
    """Causal grouped-query attention of the step's queries ``[n_tokens, n_q, d]`` over each
    sequence's cached keys and values (the new tokens' own are already written).  ``sink``: one more term in the
    softmax's denominator (a key of score 0 without a value)."""
    n_q, d = q.shape[1], q.shape[2]
    n_kv = kv.k.shape[1]
    fast = q.dtype == torch.bfloat16 and d in FAST_HEAD_DIMS and kv.page_size == 64 and n_q // n_kv <= 16
    if fast and ctx.all_single:
        if not sink and decode_flat_preferred(ctx, n_kv, kv):
            return F.attention_decode_flat(q, None, n_q, n_kv, d, None, None, 1.0, None, None, kv, ctx.kv_len, ctx.slots,
                                           ctx.max_position, scale, window)
        splits = decode_split_count(ctx, n_kv, kv)
        return F.attention_decode(q, kv, ctx.kv_len, ctx.slots, scale, window, splits, sink=sink)
    if fast:
        return F.attention_prefill(q, kv, ctx.cu_q, ctx.kv_len, ctx.slots, ctx.max_q_len, scale, window, sink=sink)
    return F.attention_exact(q, kv, ctx.tok_pos, ctx.tok_seq, ctx.slots, scale, window, sink=sink, longest_run=ctx.max_q_len)


# "0" sends bfloat16 latent attention through the exact kernel too (for measurements and for telling the kernels apart)
LATENT_TILED = os.environ.get("GTAR_B200_LATENT_TILED", "1") != "0"


def latent_attention(q_carried: torch.Tensor, q_raw: torch.Tensor, q_rot_at: int, rot: int, rot_dims: int, cos, sin,
                     cache: F.PagedRows, ctx, scale: float, window: int, out: torch.Tensor) -> torch.Tensor:
    """Attention of the step's queries over each sequence's cached latent rows (the new tokens' own are already
    written): ``q_carried [n_tokens, n_heads, rank]`` is the unrotated query carried into the latent, ``q_raw`` holds
    each head's own part to rotate at ``q_rot_at``; ``out [n_tokens, n_heads, rank]`` is the weighted sum of latents."""
    if LATENT_TILED and q_raw.dtype == torch.bfloat16 and F.latent_tiled_ok(q_carried.shape[1], q_carried.shape[2], rot, cache):
        splits = 1
        if ctx.all_single:
            splits = F.latent_splits(ctx.n_seqs, q_carried.shape[1], ctx.typical_kv_len or ctx.max_kv_len, window,
                                     F.sm_count(q_raw.device))
        return F.attention_latent_tiled(q_carried, q_raw, q_rot_at, rot, rot_dims, cos, sin, cache, ctx.tok_pos, ctx.cu_q,
                                        ctx.slots, scale, window, out, ctx.n_seqs, ctx.max_q_len, splits)
    return F.attention_latent_exact(q_carried, q_raw, q_rot_at, rot, rot_dims, cos, sin, cache, ctx.tok_pos, ctx.tok_seq,
                                    ctx.slots, scale, window, out)
