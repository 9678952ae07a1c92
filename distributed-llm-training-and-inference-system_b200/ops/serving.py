"""Serving ops: paged KV append (K13), paged decode attention (K12), batched sampling (K14).  CUDA/bf16 runs
the native kernels; CPU tensors run a plain PyTorch restatement (used by the CPU tests and as the oracle)."""
from __future__ import annotations

import math
from functools import lru_cache
from typing import Optional

import torch

from . import native

c_void_p, c_int, c_ll, c_float = native.c_void_p, native.c_int, native.c_ll, native.c_float
native.register_signature("llmctl_kv_append", [c_void_p, c_ll, c_int, c_int, c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p])
native.register_signature("llmctl_paged_attn_decode",
                          [c_void_p, c_ll, c_void_p, c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_ll, c_void_p,
                           c_int, c_int, c_int, c_int, c_int, c_int, c_float, c_void_p])
native.register_signature("llmctl_paged_attn_scratch_elems", [c_int, c_int, c_int, c_int], restype=c_ll)
native.register_signature("llmctl_sample", [c_void_p, c_int, c_ll, c_int, c_int] + [c_void_p] * 6 + [c_void_p])


def _check(ok: bool, what: str) -> None:
    if not ok:
        raise ValueError(what)


def _check_cache(cache: torch.Tensor, like: torch.Tensor, row: int) -> None:
    _check(cache.is_cuda and cache.dtype == like.dtype and cache.is_contiguous() and cache.data_ptr() % 16 == 0 and cache.numel() % row == 0,
           f"a cache is contiguous rows of {row} {like.dtype} numbers on the GPU, from a 16-byte boundary")


def kv_append(qkv: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, slot_mapping: torch.Tensor,
              heads: int, head_dim: int) -> None:
    """qkv: [T, 3*heads*head_dim] (post-RoPE); caches: [blocks, block_size, heads, head_dim];
    slot_mapping: int64 [T] (negative = skip)."""
    hd = heads * head_dim
    if qkv.is_cuda:
        if native.fast.kv_append(qkv, k_cache, v_cache, slot_mapping, heads, head_dim) is not None:
            return
        _check(qkv.dim() == 2 and qkv.dtype.itemsize == 2 and qkv.shape[1] >= 3 * hd > 0, f"qkv: 16-bit rows of at least {3 * hd} numbers")
        _check_cache(k_cache, qkv, hd)
        _check_cache(v_cache, qkv, hd)
        _check(slot_mapping.is_cuda and slot_mapping.dtype == torch.int64 and slot_mapping.numel() >= qkv.shape[0], "slot_mapping: int64 on the GPU, one per row")
        slot_mapping = slot_mapping.contiguous()
        if qkv.stride(1) != 1 or qkv.data_ptr() % 16:
            qkv = qkv.clone(memory_format=torch.contiguous_format)
        native.call("llmctl_kv_append", qkv.data_ptr(), qkv.stride(0), hd, 2 * hd, k_cache.data_ptr(),
                    v_cache.data_ptr(), slot_mapping.data_ptr(), qkv.shape[0], heads, head_dim, native.stream_ptr())
        return
    ok = slot_mapping >= 0
    kc, vc = k_cache.view(-1, hd), v_cache.view(-1, hd)
    kc[slot_mapping[ok]] = qkv[ok, hd:2 * hd]
    vc[slot_mapping[ok]] = qkv[ok, 2 * hd:3 * hd]


def choose_splits(batch: int, heads: int, max_context: int, block_size: int, sms: int = 148) -> int:
    # Each CTA walks block table -> K/V rows -> online softmax in a dependent chain, so HBM fills up with a few CTAs per SM and many more
    # to follow.  Splits are whole KV blocks of >= 64 tokens; the merge pass costs (head_dim + 2) floats per split, ~3 % of the K/V bytes at
    # 64 tokens per split.
    # Up to 512 (head, sequence) pairs a CTA walks at most 512 tokens where 8 splits allow it; more pairs fill the waves by themselves, and
    # what each split adds is lost.  Around the line the splits differ by 2% either way (us by splits, contexts from a quarter of the stated
    # one: 16 sequences of up to 4096, 32 heads of 128 2: 109.0, 8: 110.8, 16: 118.0; 32 of them 2: 200.1, 8: 203.3; 64 1: 374.6, 4: 383.5; 256 of up
    # to 1500 1: 551.7, 4: 575.2; 64 of up to 2304, 12 heads of 64 1: 55.3, 2: 53.9, 8: 54.3); it was drawn for a kernel that took a quarter
    # longer, whose full batches of unlike contexts gained 10% by 8 splits.
    want = max(1, (8 * sms + batch * heads - 1) // (batch * heads), min(8, (max_context + 511) // 512) if batch * heads <= 512 else 1)
    per_split = max(block_size, (64 // block_size) * block_size) if block_size <= 64 else block_size
    return int(max(1, min(want, max(1, max_context // per_split), 256)))


@lru_cache(maxsize=4096)
def _launch_splits(batch: int, heads: int, head_dim: int, max_context: int, block_size: int, sms: int = 148) -> int:
    # One launch, merged inside clusters of up to 8 splits, while all CTAs (three per SM) are resident together and none walks
    # more than 768 tokens (us in one launch / in the splits of choose_splits with a merge kernel: one context of 4096, 32 heads of 128
    # 14.5 in 8 / 16.8 in 16; 8 of up to 2304, 4 heads 13.5 / 13.8; 64 of 500, 4 heads 12.6 / 12.3).  Beyond one
    # wave a single split without a merge kernel pays for the shortest walks only (64 of 500, 12 heads of 64: 13.5 / 14.8; 32 heads of
    # 128: 65.1 / 62.8); larger batches and longer contexts take choose_splits.
    resident = min(8, 3 * sms // (batch * heads))
    if max_context <= 768 * resident:
        return max(1, min(resident, max_context // 64))
    if resident == 0 and max_context * head_dim <= 512 * 64:
        return 1
    return choose_splits(batch, heads, max_context, block_size, sms)


def paged_attention_decode(q: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor,
                           block_tables: torch.Tensor, context_lens: torch.Tensor, max_context: int,
                           scale: Optional[float] = None, num_splits: Optional[int] = None,
                           scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
    """q: [B, heads, head_dim]; block_tables: int32 [B, max_blocks]; context_lens: int32 [B] -> [B, heads, head_dim]."""
    B, H, D = q.shape
    block_size = k_cache.shape[1]
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if q.is_cuda:
        ns = num_splits or _launch_splits(B, H, D, max_context, block_size)
        if scratch is None:
            out = native.fast.paged_decode(q, k_cache, v_cache, block_tables, context_lens, max_context, ns, scale)
            if out is not None:
                return out
        _check(q.dtype == torch.bfloat16, "q: bfloat16")
        _check_cache(k_cache, q, H * D)
        _check_cache(v_cache, q, H * D)
        _check(k_cache.shape == v_cache.shape, "k_cache and v_cache: of one shape")
        _check(block_tables.is_cuda and block_tables.dtype == torch.int32 and block_tables.dim() == 2 and block_tables.shape[0] >= B,
               "block_tables: int32 on the GPU, a row per sequence")
        _check(context_lens.is_cuda and context_lens.dtype == torch.int32 and context_lens.numel() >= B, "context_lens: int32 on the GPU, one per sequence")
        block_tables, context_lens = block_tables.contiguous(), context_lens.contiguous()
        if q.stride(2) != 1 or q.stride(1) != D or q.data_ptr() % 16:
            q = q.clone(memory_format=torch.contiguous_format)
        need = native.lib().llmctl_paged_attn_scratch_elems(B, H, D, ns)
        if need and (scratch is None or scratch.numel() < need or scratch.dtype != torch.float32 or not scratch.is_contiguous()):
            scratch = torch.empty(need, dtype=torch.float32, device=q.device)
        out = torch.empty(B, H, D, dtype=q.dtype, device=q.device)
        native.call("llmctl_paged_attn_decode", q.data_ptr(), q.stride(0), k_cache.data_ptr(), v_cache.data_ptr(),
                    block_tables.data_ptr(), block_tables.shape[1], context_lens.data_ptr(), out.data_ptr(),
                    out.stride(0), native.ptr(scratch), B, H, D, block_size, int(max_context), ns, float(scale),
                    native.stream_ptr())
        if need:
            native.count_launches(1)        # the merge kernel
        return out
    out = torch.zeros(B, H, D, dtype=q.dtype)
    for b in range(B):
        n = int(context_lens[b])
        if n == 0:
            continue
        idx = torch.arange(n)
        slots = block_tables[b, idx // block_size].long() * block_size + idx % block_size
        k = k_cache.view(-1, H, D)[slots].float()
        v = v_cache.view(-1, H, D)[slots].float()
        s = torch.einsum("hd,nhd->hn", q[b].float(), k) * scale
        out[b] = torch.einsum("hn,nhd->hd", torch.softmax(s, -1), v).to(q.dtype)
    return out


def sample_reference(logits: torch.Tensor, temperature: float, top_k: int, top_p: float,
                     generator: Optional[torch.Generator] = None) -> int:
    """The reference's sampling pipeline for one row (reference llmctl/serve/server.py:209-235), restated."""
    x = logits.float().clone()      # never edit the caller's logits
    if temperature <= 0:
        return int(x.argmax())
    if temperature != 1.0:
        x = x / temperature
    if top_k and top_k > 0:
        kth = torch.topk(x, min(top_k, x.numel())).values[-1]
        x = torch.where(x < kth, torch.full_like(x, float("-inf")), x)
    if top_p < 1.0:
        sx, si = torch.sort(x, descending=True)
        cp = torch.softmax(sx, -1).cumsum(-1)
        remove = cp > top_p
        remove[1:] = remove[:-1].clone()
        remove[0] = False
        x[si[remove]] = float("-inf")
    return int(torch.multinomial(torch.softmax(x, -1), 1, generator=generator))


def sample(logits: torch.Tensor, temperature: torch.Tensor, top_k: torch.Tensor, top_p: torch.Tensor,
           uniform: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Batched sampling.  logits [B, V] bf16/fp32; per-row parameter tensors; returns int64 [B]."""
    B, V = logits.shape
    if logits.is_cuda:
        if uniform is None:
            uniform = torch.rand(B, device=logits.device)
        out = torch.empty(B, dtype=torch.int64, device=logits.device)
        native.call("llmctl_sample", logits.data_ptr(), int(logits.dtype == torch.float32), logits.stride(0), B, V,
                    temperature.data_ptr(), top_k.data_ptr(), top_p.data_ptr(), uniform.data_ptr(), out.data_ptr(),
                    None, native.stream_ptr())
        return out
    return torch.tensor([sample_reference(logits[i], float(temperature[i]), int(top_k[i]), float(top_p[i]))
                         for i in range(B)], dtype=torch.int64)
