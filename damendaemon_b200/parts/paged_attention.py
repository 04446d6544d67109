"""Paged causal attention of a step's tokens: the cache write and the choice of kernel.

Seven kernels can serve (csrc/attention_*.cu): the general one (any sizes, both dtypes: the fallback and the
reference of the others; the mma.sync prompt kernel takes the portions of other head sizes in padded
tiles), one for single tokens of either dtype (whole rows on the CUDA cores), a float32 prompt kernel, two bfloat16 decode kernels (rows by cp.async; whole pages of a group of
heads by TMA) and two bfloat16 prompt kernels (mma.sync; tcgen05). Which one a step takes depends on the step
(decode only or not, how many (token, head) pairs), on what each kernel supports (head size, page size, groups) and
on thresholds that were measured, which are data: ``AttentionTuning``, a field of the runtime, not constants of a
model. A mixer calls ``paged_attention`` through ``ctx.attend``.
"""
from __future__ import annotations

from dataclasses import dataclass

import torch

from .. import kernels

PAGES_HEAD_DIM = 64                       # the only head size of the page-streaming decode kernel


@dataclass(frozen=True)
class AttentionTuning:
    """Thresholds of the kernel choice. Whole pages by TMA are ahead of rows at any number of single tokens (us a layer of a
    whole decode step on a B200, rows / pages: 25 heads, one request at 64, 300, 600, 900 keys 31.3 / 28.5, 31.3 / 29.7,
    31.2 / 30.4, 31.6 / 31.6; two at 900 34.9 / 32.9, four at 540 37.2 / 33.6; 16 heads, eight at 900
    37.9 / 33.0; one request of 4,000 keys in a table of 4,096 42.3 / 38.7), so by default every step takes them. The
    splits are dealt out by the contexts (attention_decode_pages_splits): cut by row_keys_per_block instead, four requests at
    900 keys x 25 heads took 42.0 us and eight at 900 x 16 heads 40.7 (now 35.5 and 33.0)."""
    pages_from_pairs: int = 1             # steps with at least this many (token, head) pairs stream whole pages,
    pages_from_pair_keys: int = 200_000   # ... or with this many pairs x keys of context; others take the row kernel
    row_keys_per_block: int = 128         # key split of the row decode kernel: keys per block ...
    row_blocks_per_sm: int = 2            # ... and blocks wanted per SM


def prompt_key_block(n_heads, kv_heads, head_dim, page_size, dtype):
    """Where the tcgen05 prompt kernel likes prompts to be cut, or 1 if it does not take these sizes: a portion that
    starts on a key block lets the kernel write the cache itself and read whole blocks."""
    if kernels.attention_prefill_tcgen05_supported(n_heads, kv_heads, head_dim, page_size, dtype):
        return kernels.ATTENTION_PREFILL_TCGEN05_KEY_BLOCK
    return 1


def paged_attention(ctx, q, k, v, cache, n_heads, scale, window=None, chunk=None, gate=None, value_dim=None, keep_first=0,
                    softcap=None, sink=None, exact_weights=False):
    runtime = ctx.runtime
    tune = runtime.attention_tuning
    if (k is None) != (v is None) or (k is None and cache.writable):
        raise ValueError("keys and values come together; only a mixer that reads another stop's cache brings none")
    if k is None:
        # queries only: the keys and values are another stop's, in the cache already
        if q.stride(1) != 1 or (gate is not None and (gate.stride(0) != q.stride(0) or gate.stride(1) != 1)):
            q = q.contiguous()
            gate = None if gate is None else gate.contiguous()
    elif not (q.stride(0) == k.stride(0) == v.stride(0)) or q.stride(1) != 1 or k.stride(1) != 1 or v.stride(1) != 1 or \
            (gate is not None and (gate.stride(0) != q.stride(0) or gate.stride(1) != 1)):
        # the kernels read q, k and v as row views of one buffer (what a fused projection leaves); a part that made
        # new tensors of some of them (a position encoding that does not rotate in place) gets them packed again
        parts = [q, k, v] + ([gate] if gate is not None else [])
        packed = torch.cat(parts, dim=1).split([p.shape[1] for p in parts], dim=1)
        q, k, v = packed[:3]
        gate = packed[3] if gate is not None else None
    kv, table = cache.kv, ctx.block_table(cache.group)
    keep_first = keep_first if window is not None or chunk is not None else 0
    # first keys kept behind the window, capped scores, a sink in the softmax: the general kernel, the row decode kernel and
    # the mma.sync prompt kernel take them; the latter two also the weights in two bfloat16 terms (the general kernel's are
    # float32 anyway)
    more = dict(keep_first=keep_first, softcap=softcap, sink=sink)
    special = bool(keep_first or softcap or sink is not None or exact_weights)
    exact = dict(more, exact_weights=exact_weights) if special else {}
    if value_dim is not None and value_dim != cache.group.need.head_dim:
        need = cache.group.need
        # value heads of their own size: kernels that are told the page's geometry
        if cache.writable:
            kernels.kv_store(k, v, ctx.token_entry, ctx.positions, table, kv, kv_heads=need.kv_heads, head_dim=need.head_dim,
                             v_dim=value_dim)
        return general_attention(ctx, q, kv, table, n_heads, scale, window, need.kv_heads, need.head_dim, value_dim, exact_weights,
                                 chunk=chunk, gate=gate, **more)
    kv_heads, page_size, head_dim = kv.shape[2], kv.shape[3], kv.shape[4]
    k_new, v_new = (k, v) if cache.writable else (None, None)
    fast = runtime.attention != "rows"
    masked = dict(chunk=chunk, gate=gate)      # every kernel takes the chunked mask and the gate on its output
    # the kernels that read whole rows on the CUDA cores (CUDA tensors only: they ask for the rows' alignment). For float32 they
    # serve every step; in bfloat16 one of them takes the single tokens of the sizes that the tensor-core decode kernels refuse
    def cores():
        return q.is_cuda and fast and not special and kernels.attention_cores_supported(q, kv, k_new, v_new)
    if q.dtype == torch.float32 and cores():
        return float32_attention(ctx, q, k_new, v_new, kv, table, n_heads, scale, window, **masked)
    tensor = fast and runtime.attention != "mma" and not special
    # a sink alone (no kept first keys, no cap, no weights in two terms) the tcgen05 prompt kernel takes as well
    sink_only = sink is not None and not (keep_first or softcap or exact_weights)
    def decode_splits(n_tokens):
        """(kernel, pieces of a token's keys) for single tokens that a tensor-core decode kernel takes."""
        pairs = n_tokens * n_heads
        # (the kernels are asked only about the head size that pages can have: an eager step asks for every layer)
        many = pairs >= tune.pages_from_pairs or pairs * ctx.split_context >= tune.pages_from_pair_keys
        if tensor and many and head_dim == PAGES_HEAD_DIM and \
                kernels.attention_decode_pages_supported(n_heads, kv_heads, head_dim, page_size, q.dtype):
            # whole pages of a group of heads by TMA
            return "pages", kernels.attention_decode_pages_splits(n_tokens, n_heads, page_size, ctx.split_context, q.device)
        if kernels.attention_decode_supported(n_heads, kv_heads, head_dim, q.dtype):
            return "rows", ctx.key_splits(n_heads, keys_per_block=tune.row_keys_per_block, blocks_per_sm=tune.row_blocks_per_sm, n_tokens=n_tokens)
        return None, 0
    if ctx.decode_only and fast:
        kernel, splits = decode_splits(ctx.n_tokens)
        if kernel:
            # the decode kernels take the new keys and values from the projection and write them (decode only: token t is entry t,
            # so they are spared the look-up)
            return kernels.attention_decode(q, kv, None, ctx.positions, table, n_heads, scale, window,
                                            n_splits=splits, k_new=k_new, v_new=v_new, kernel=kernel, **masked, **exact)
    # key/value groups and small heads (8 requests x 25 heads on 5, 400 keys: 9 us, 32 through the general kernel and the cache
    # write; 32 x 16 on 4, 600 keys: 37 / 69; 8 x 32 heads of 128 on 8: 32 / 41)
    if ctx.decode_only and tensor and cores():
        return kernels.attention_tokens(q, kv, ctx.positions, table, n_heads, scale, window, n_splits=token_splits(ctx, ctx.n_tokens, n_heads),
                                        k_new=k_new, v_new=v_new, **masked)
    tcgen05 = not ctx.decode_only and (tensor or (sink_only and fast and runtime.attention != "mma")) and \
        kernels.attention_prefill_tcgen05_supported(n_heads, kv_heads, head_dim, page_size, q.dtype)
    mma = not tcgen05 and not ctx.decode_only and fast and kernels.attention_prefill_supported(n_heads, kv_heads, head_dim, q.dtype)
    # A step that mixes portions with single tokens: the single tokens come first (ctx.n_single) and go to a decode
    # kernel, the portions to a prompt kernel. A prompt kernel spends a tile of 64 or 128 query rows and a walk over all
    # key blocks on a single token (measured with 56 decoding requests beside 8 portions of 249 tokens, 36 layers:
    # 8.3 ms a step through the prompt kernel alone, against 4.5 ms for 2,048 prompt tokens).
    n1 = ctx.n_single if tcgen05 or mma else 0
    kernel, splits = decode_splits(n1) if n1 and kernels.attention_decode_supported(n_heads, kv_heads, head_dim, q.dtype) else (None, 0)
    if n1 and not kernel and not (tensor and cores()):
        n1 = 0
    out = None
    if n1:
        out = torch.empty((q.shape[0], n_heads * head_dim), dtype=q.dtype, device=q.device)
        if not kernel:
            kernels.attention_tokens(q[:n1], kv, ctx.positions[:n1], table, n_heads, scale, window, n_splits=token_splits(ctx, n1, n_heads),
                                     out=out[:n1], k_new=None if k_new is None else k_new[:n1], v_new=None if v_new is None else v_new[:n1],
                                     chunk=chunk, gate=None if gate is None else gate[:n1])
        else:
            kernels.attention_decode(q[:n1], kv, None, ctx.positions[:n1], table, n_heads, scale, window, n_splits=splits,
                                     out=out[:n1], k_new=None if k_new is None else k_new[:n1],
                                     v_new=None if v_new is None else v_new[:n1], kernel=kernel,
                                     chunk=chunk, gate=None if gate is None else gate[:n1], **exact)
        if n1 == ctx.n_entries:
            return out
    # the tcgen05 prompt kernel writes the cache itself when no key block of its entries mixes cached and new keys
    fused_store = tcgen05 and cache.writable and ctx.aligned_starts and n1 == ctx.n_single
    if cache.writable and not fused_store:
        kernels.kv_store(k[n1:], v[n1:], ctx.token_entry[n1:], ctx.positions[n1:], table, kv)
    if tcgen05:
        return kernels.attention_prefill(q, kv, ctx.entry_start[n1:], ctx.entry_pos0[n1:], table[n1:], n_heads, scale, window,
                                         out=out, kernel="tcgen05", k_new=k_new, v_new=v_new, store_new=fused_store,
                                         **({} if sink is None else {"sink": sink}), **masked)
    if mma:
        return kernels.attention_prefill(q, kv, ctx.entry_start[n1:], ctx.entry_pos0[n1:], table[n1:], n_heads, scale, window,
                                         out=out, **masked, **exact)
    return general_attention(ctx, q, kv, table, n_heads, scale, window, kv_heads, head_dim, head_dim, exact_weights, chunk=chunk,
                             gate=gate, **(more if special else {}))


def float32_attention(ctx, q, k_new, v_new, kv, table, n_heads, scale, window, chunk, gate):
    """A float32 cache: single tokens (which lie first) go to the kernel that reads whole rows and writes their own key and
    value, portions to the one that shares key blocks among 64 queries."""
    n1 = ctx.n_entries if ctx.decode_only else ctx.n_single
    if n1 == q.shape[0]:
        return kernels.attention_tokens(q, kv, ctx.positions, table, n_heads, scale, window, n_splits=token_splits(ctx, n1, n_heads),
                                            k_new=k_new, v_new=v_new, chunk=chunk, gate=gate)
    out = torch.empty_like(q, memory_format=torch.contiguous_format)
    if k_new is not None:
        kernels.kv_store(k_new[n1:], v_new[n1:], ctx.token_entry[n1:], ctx.positions[n1:], table, kv)
    if n1:
        kernels.attention_tokens(q[:n1], kv, ctx.positions[:n1], table, n_heads, scale, window, n_splits=token_splits(ctx, n1, n_heads),
                                     out=out[:n1], k_new=None if k_new is None else k_new[:n1], v_new=None if v_new is None else v_new[:n1],
                                     chunk=chunk, gate=None if gate is None else gate[:n1])
    # A tile's keys are shared among blocks while tiles x heads leave SMs without their three blocks: few in all, or long
    # portions whose last tiles work longest (us in 1 / 2 / 4 pieces: 32 queries x 2 heads at 100 keys 25 / 19 / 13, 200 x 4
    # 46 / 27 / 18; 1,000 x 20 135 / 111 / 135; but 2 x 1,024 x 25 255 / 266 / 322, and 8 prompts of 64 x 25, whose tiles have
    # one block of keys, 14 / 25 / 43).
    n, entries = q.shape[0] - n1, ctx.n_entries - n1
    blocks = (-(-n // 64) + entries - 1) * n_heads
    splits = 4 if 4 * blocks <= 3 * ctx.sm_count else (2 if 2 * blocks <= 5 * ctx.sm_count and n >= 128 * entries else 1)
    return kernels.attention_f32_prompt(q, kv, ctx.entry_start[n1:], ctx.entry_pos0[n1:], table[n1:], n_heads, scale, window, out=out,
                                        n_splits=min(splits, max(1, ctx.split_context // 128)), chunk=chunk, gate=gate)


def token_splits(ctx, n_tokens, n_heads, keys_per_block=128):
    """Blocks that share a token's keys: as many as are resident at once (two an SM; a second wave costs more than longer
    pieces: 200 (token, head) pairs of 70 keys in one and in two pieces 5.6 and 10.9 us), each with at least half a round of
    its eight warps, and at most four but for long contexts (us in 1 / 2 / 4 / 8 pieces, bfloat16, 25 pairs on 5 heads: 1,000
    keys 7.8 / 5.2 / 4.3 / 4.8, 16,000 keys 140 / 77 / 42 / 24; 128 pairs of 128 on 32, 16,000 keys 328 / 188 / 193 / 197)."""
    want = 2 * ctx.sm_count // max(1, n_tokens * n_heads)
    return max(1, min(want, -(-ctx.split_context // keys_per_block), 4 if ctx.split_context <= 4096 else 8))


def general_attention(ctx, q, kv, table, n_heads, scale, window, kv_heads, head_dim, value_dim, exact_weights=False, gate=None, **mask):
    """Head sizes that have no kernel of their own, the keys and values in the cache already: the general kernel; for a step with
    portions in bfloat16 its single tokens only (cut into splits of the keys), the portions on the tensor cores in tiles padded
    to the next size, where the sizes allow it."""
    runtime = ctx.runtime
    sizes = {} if value_dim == head_dim else dict(kv_heads=kv_heads, v_dim=value_dim)
    if ctx.decode_only or runtime.attention == "rows" or \
            not kernels.attention_prefill_padded_supported(n_heads, kv_heads, head_dim, value_dim, q.dtype):
        return kernels.attention_rows(q, kv, ctx.token_entry, ctx.positions, table, n_heads, scale, window,
                                      n_splits=ctx.key_splits(n_heads), gate=gate, **mask, **sizes)
    out = torch.empty((q.shape[0], n_heads * value_dim), dtype=q.dtype, device=q.device)
    n1 = ctx.n_single
    if n1:
        kernels.attention_rows(q[:n1], kv, ctx.token_entry[:n1], ctx.positions[:n1], table, n_heads, scale, window, out=out[:n1],
                               n_splits=ctx.key_splits(n_heads, n_tokens=n1), gate=None if gate is None else gate[:n1], **mask, **sizes)
    if n1 < ctx.n_entries:
        kernels.attention_prefill_padded(q, kv, ctx.entry_start[n1:], ctx.entry_pos0[n1:], table[n1:], n_heads, scale, window, out=out,
                                         gate=gate, exact_weights=exact_weights, **mask, **sizes)
    return out
