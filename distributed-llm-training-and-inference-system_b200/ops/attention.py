"""Causal attention front-end (K6).

``attention(q, k, v)`` takes ``[B, S, H, D]`` views (typically slices of the packed qkv activation) and
dispatches to the tcgen05 flash-attention kernels (``csrc/attention``) when they are built and the shape is
supported (bf16, head_dim 64 or 128; causal sequences of any length, others of whole 128-token tiles), else to PyTorch
SDPA (other head sizes, non-causal ragged shapes, CPU).

Reference: the reference never calls attention itself — HF modules pick SDPA/eager behind
``self.model(**batch)`` (reference llmctl/runtime/engine.py:284); its tuner benchmarks a naive
softmax(QK^T)V (reference llmctl/plugins/autotuning.py:149-188).
"""
from __future__ import annotations

import math
from typing import Optional

import torch
import torch.nn.functional as F

from . import native
from .functional import _whole_units, kernel_config

c_void_p, c_int, c_ll, c_float = native.c_void_p, native.c_int, native.c_ll, native.c_float

native.register_signature(
    "llmctl_flash_attn_fwd",
    [c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,  # q k v o lse
     c_int, c_int, c_int, c_int,                         # B S H D
     c_ll, c_ll, c_ll, c_ll,                             # q_row_stride k_row_stride v_row_stride o_row_stride (elements per token)
     c_float, c_int, c_void_p])                          # scale causal stream
native.register_signature(
    "llmctl_flash_attn_bwd",
    [c_void_p] * 10 +                                    # q k v o do lse dq dk dv scratch
    [c_int, c_int, c_int, c_int] + [c_ll] * 5 + [c_float, c_int, c_void_p])


def _native_built(q: torch.Tensor) -> bool:
    return (q.is_cuda and q.dtype == torch.bfloat16 and kernel_config().attention == "native"
            and native.has_symbol("llmctl_flash_attn_fwd"))


def _native_shape(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal: bool) -> bool:
    """The kernels' tiles end inside a sequence only under the causal mask, which hides the keys past its end."""
    return q.shape[-1] in (64, 128) and (causal or q.shape[1] % 128 == 0) and k.shape == q.shape and v.shape == q.shape


def _native_ok(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal: bool = True) -> bool:
    """The kernels read these views where they lie: heads side by side in a token, whole 16-byte units, sequences back to back."""
    return _native_built(q) and _native_shape(q, k, v, causal) and _native_layout(q, k, v)


def _native_layout(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> bool:
    B, S, H, D = q.shape
    for t in (q, k, v):
        if (t.dtype != q.dtype or t.stride(3) != 1 or t.stride(2) != D or (B > 1 and t.stride(0) != S * t.stride(1))
                or t.stride(1) % 8 or t.data_ptr() % 16):
            return False
    return True


def _stats_scratch(B: int, S: int, H: int, device: torch.device) -> torch.Tensor:
    """Scratch of the backward: two numbers per (head, query), sequences rounded up to whole tiles, and the item counter (in two words)."""
    return torch.empty(2 * B * H * ((S + 127) // 128 * 128) + 2, dtype=torch.float32, device=device)


class _FlashAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, scale, causal):
        B, S, H, D = q.shape
        o = torch.empty(B, S, H, D, dtype=q.dtype, device=q.device)
        lse = torch.empty(B, H, S, dtype=torch.float32, device=q.device)
        native.call("llmctl_flash_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(),
                    B, S, H, D, q.stride(1), k.stride(1), v.stride(1), o.stride(1), float(scale), int(causal),
                    native.stream_ptr())
        native.keep(ctx, q, k, v, o, lse)
        ctx.scale, ctx.causal = scale, causal
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = native.kept(ctx)
        if native.has_symbol("llmctl_flash_attn_bwd"):
            B, S, H, D = q.shape
            if not _native_layout(q, k, v):
                q, k, v = (t.clone(memory_format=torch.contiguous_format) for t in (q, k, v))
            o, lse, do = _whole_units(o), _whole_units(lse), _whole_units(do)
            # dq|dk|dv packed like the forward's qkv so the following wgrad GEMM sees one tensor
            dqkv = torch.empty(B, S, 3, H, D, dtype=q.dtype, device=q.device)
            dq, dk, dv = dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2]
            scratch = _stats_scratch(B, S, H, q.device)
            native.call("llmctl_flash_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                        do.data_ptr(), lse.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                        scratch.data_ptr(), B, S, H, D, q.stride(1), k.stride(1), v.stride(1), o.stride(1),
                        dq.stride(1), float(ctx.scale), int(ctx.causal), native.stream_ptr())
            return dq, dk, dv, None, None
        # backward not built yet: recompute through SDPA (library path) for the gradient only
        with torch.enable_grad():
            qq, kk, vv = (t.detach().requires_grad_(True) for t in (q, k, v))
            out = _sdpa(qq, kk, vv, ctx.causal, ctx.scale)
            dq, dk, dv = torch.autograd.grad(out, (qq, kk, vv), do)
        return dq, dk, dv, None, None


def _sdpa(q, k, v, causal, scale):
    o = F.scaled_dot_product_attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2),
                                       is_causal=causal, scale=scale)
    return o.transpose(1, 2)


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, causal: bool = True,
              scale: Optional[float] = None) -> torch.Tensor:
    scale = scale if scale is not None else 1.0 / math.sqrt(q.shape[-1])
    if kernel_config().attention == "native":
        o = native.fast.attention(q, k, v, scale, causal)
        if o is not None:
            return o
    if _native_ok(q, k, v, causal):
        return native.apply(_FlashAttnFn, q, k, v, scale, causal)
    if (_native_built(q) and _native_shape(q, k, v, causal) and k.dtype == v.dtype == q.dtype
            and (q.shape[-1] == 64 or q.shape[1] % 128 or any(t.data_ptr() % 16 for t in (q, k, v)))):
        # other strides: head_dim 64 and ragged lengths (gpt-125m, every serving prefill) are always copied for the kernel, whole
        # 128-wide tiles are left to the library.  Odd addresses are always copied: the library reads 16-byte units as well.
        q, k, v = (t.clone(memory_format=torch.contiguous_format) for t in (q, k, v))
        return native.apply(_FlashAttnFn, q, k, v, scale, causal)
    return _sdpa(q, k, v, causal, scale)


# ------------------------------------------------------------------------------------------------------
# Packed RoPE + attention: one autograd node over the packed [tokens, 3*H*D] activation.
# Slicing q/k/v out of the packed tensor through autograd costs three zero-fills, three copies and two adds
# of the full activation in backward; here the backward writes dq|dk|dv straight into one packed buffer and
# applies the inverse rotation in place on it.
# ------------------------------------------------------------------------------------------------------
_sdpa_impl = {"name": None}


def _sdpa_fwd_bwd_ops():
    """Pick the library attention op pair once (cudnn flash on sm_100, else flash-attn 2)."""
    if _sdpa_impl["name"] is None:
        _sdpa_impl["name"] = "cudnn"
    return _sdpa_impl["name"]


def _lib_attention_fwd(q, k, v, scale, causal):
    """q,k,v: [B,H,S,D] views.  Returns (out [B,H,S,D], saved-for-backward tuple)."""
    impl = _sdpa_fwd_bwd_ops()
    if impl == "cudnn":
        try:
            r = torch.ops.aten._scaled_dot_product_cudnn_attention(q, k, v, None, True, 0.0, causal, False, scale=scale)
            return r[0], ("cudnn",) + tuple(r[1:8])
        except Exception:  # noqa: BLE001
            _sdpa_impl["name"] = impl = "flash"
    if impl == "flash":
        r = torch.ops.aten._scaled_dot_product_flash_attention(q, k, v, 0.0, causal, False, scale=scale)
        return r[0], ("flash",) + tuple(r[1:8])
    raise RuntimeError("no library attention op available")


def _lib_attention_bwd(do, q, k, v, out, saved, scale, causal):
    kind = saved[0]
    lse, cq, ck, mq, mk, seed, off = saved[1:8]
    if kind == "cudnn":
        bias = torch.empty(0, device=q.device, dtype=q.dtype)
        try:
            return torch.ops.aten._scaled_dot_product_cudnn_attention_backward(
                do, q, k, v, out, lse, seed, off, None, cq, ck, mq, mk, 0.0, causal, scale=scale)
        except Exception:  # noqa: BLE001
            return torch.ops.aten._scaled_dot_product_cudnn_attention_backward(
                do, q, k, v, out, lse, seed, off, bias, cq, ck, mq, mk, 0.0, causal, scale=scale)
    return torch.ops.aten._scaled_dot_product_flash_attention_backward(
        do, q, k, v, out, lse, cq, ck, mq, mk, 0.0, causal, seed, off, scale=scale)


class _RopeAttnPackedFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, cos, sin, B, S, H, D, positions, scale, use_native):
        T = B * S
        # RoPE in place on the q and k heads (the producing GEMM does not keep its output)
        native.call("llmctl_rope_inplace", qkv.data_ptr(), qkv.stride(0), T, 2 * H, D, cos.data_ptr(), sin.data_ptr(),
                    native.ptr(positions), S, 1.0, native.stream_ptr())
        v5 = qkv.detach().view(B, S, 3, H, D)
        q, k, v = v5[:, :, 0], v5[:, :, 1], v5[:, :, 2]
        if use_native:
            o = torch.empty(B, S, H, D, dtype=qkv.dtype, device=qkv.device)
            lse = torch.empty(B, H, S, dtype=torch.float32, device=qkv.device)
            native.call("llmctl_flash_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(),
                        B, S, H, D, q.stride(1), k.stride(1), v.stride(1), o.stride(1), float(scale), 1,
                        native.stream_ptr())
            ctx.lib_saved = None
            native.keep(ctx, qkv.detach(), o, lse, cos, sin, positions if positions is not None else torch.empty(0))
            out = o
        else:
            o_bhsd, saved = _lib_attention_fwd(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), scale, True)
            ctx.lib_saved = (saved[0],) + tuple(x for x in saved[1:])
            native.keep(ctx, qkv.detach(), o_bhsd, saved[1], cos, sin,
                                  positions if positions is not None else torch.empty(0))
            out = o_bhsd.transpose(1, 2)
        ctx.meta = (B, S, H, D, positions is not None, scale, use_native)
        return out.reshape(T, H * D)

    @staticmethod
    def backward(ctx, do):
        qkv, o, lse, cos, sin, positions = native.kept(ctx)
        B, S, H, D, has_pos, scale, use_native = ctx.meta
        T = B * S
        if qkv.stride(1) != 1 or qkv.stride(0) % 8 or qkv.data_ptr() % 16:
            qkv = _whole_units(qkv)
        cos, sin, positions = _whole_units(cos), _whole_units(sin), _whole_units(positions)
        v5 = qkv.view(B, S, 3, H, D)
        q, k, v = v5[:, :, 0], v5[:, :, 1], v5[:, :, 2]
        dqkv = torch.empty(T, 3 * H * D, dtype=qkv.dtype, device=qkv.device)
        d5 = dqkv.view(B, S, 3, H, D)
        do4 = do.reshape(B, S, H, D)
        if use_native and native.has_symbol("llmctl_flash_attn_bwd"):
            o, lse, do4 = _whole_units(o), _whole_units(lse), _whole_units(do4)
            scratch = _stats_scratch(B, S, H, qkv.device)
            native.call("llmctl_flash_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do4.data_ptr(),
                        lse.data_ptr(), d5[:, :, 0].data_ptr(), d5[:, :, 1].data_ptr(), d5[:, :, 2].data_ptr(),
                        scratch.data_ptr(), B, S, H, D, q.stride(1), k.stride(1), v.stride(1), o.stride(1),
                        d5.stride(1), float(scale), 1, native.stream_ptr())
        else:
            if use_native:
                # native forward, library backward: recompute the library forward to get its saved state
                o_b, saved = _lib_attention_fwd(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), scale, True)
            else:
                o_b, saved = o, ctx.lib_saved
            dq, dk, dv = _lib_attention_bwd(do4.transpose(1, 2), q.transpose(1, 2), k.transpose(1, 2),
                                            v.transpose(1, 2), o_b, saved, scale, True)
            d5[:, :, 0].copy_(dq.transpose(1, 2))
            d5[:, :, 1].copy_(dk.transpose(1, 2))
            d5[:, :, 2].copy_(dv.transpose(1, 2))
        native.call("llmctl_rope_inplace", dqkv.data_ptr(), dqkv.stride(0), T, 2 * H, D, cos.data_ptr(), sin.data_ptr(),
                    positions.data_ptr() if has_pos else None, S, -1.0, native.stream_ptr())
        return dqkv, None, None, None, None, None, None, None, None, None


def rope_attention_packed(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, batch: int, seq: int,
                          heads: int, head_dim: int, positions: Optional[torch.Tensor] = None,
                          scale: Optional[float] = None) -> torch.Tensor:
    """RoPE(q,k) + causal attention on a packed ``[batch*seq, 3*heads*head_dim]`` activation (rows are
    ``q|k|v``).  Returns ``[batch*seq, heads*head_dim]``.  CUDA/bf16 with the native element-wise kernels
    enabled uses the fused autograd node above; everything else composes the generic ops."""
    from . import functional as ops
    scale = scale if scale is not None else 1.0 / math.sqrt(head_dim)
    cfg = kernel_config()
    if cfg.elementwise == "native" and cfg.attention == "native":
        o = native.fast.rope_attention(qkv, cos, sin, None if positions is None else positions.to(torch.int32), batch, seq, heads, head_dim, scale)
        if o is not None:
            return o
    if (qkv.is_cuda and qkv.dtype == torch.bfloat16 and cfg.elementwise == "native" and qkv.dim() == 2
            and qkv.stride(1) == 1 and not qkv.is_leaf and head_dim % 16 == 0):
        v5 = qkv.view(batch, seq, 3, heads, head_dim)
        use_native = _native_ok(v5[:, :, 0], v5[:, :, 1], v5[:, :, 2]) and \
            (native.has_symbol("llmctl_flash_attn_bwd") or not torch.is_grad_enabled())
        pos = None if positions is None else positions.to(torch.int32)
        # views the kernels only take after a copy (an odd address) go through the composed
        # ops below, where attention() makes it, instead of dropping to the library inside the fused node
        paddable = (not use_native and cfg.attention == "native" and native.has_symbol("llmctl_flash_attn_bwd")
                    and (head_dim == 64 or (head_dim == 128 and (seq % 128 != 0 or qkv.data_ptr() % 16 != 0))))
        if not paddable:
            return native.apply(_RopeAttnPackedFn, qkv, cos, sin, batch, seq, heads, head_dim, pos, scale, use_native)
    qkv = ops.rope_packed(qkv, cos, sin, 2 * heads, head_dim, seq, positions)
    v5 = qkv.view(batch, seq, 3, heads, head_dim)
    o = attention(v5[:, :, 0], v5[:, :, 1], v5[:, :, 2], causal=True, scale=scale)
    return o.reshape(batch * seq, heads * head_dim)
