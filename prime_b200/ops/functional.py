"""Autograd-aware ops used by the eager modules.

CPU tensors: ordinary differentiable torch math (fp32 internally) — this is also the numerical
oracle. CUDA tensors: ``torch.autograd.Function`` wrappers whose forward and backward are the
hand-written sm_100a kernels (bf16 activations / weights, fp32 accumulation). fp32 CUDA inputs are
cast to bf16 at the op boundary, which mirrors the reference's FSDP2 mixed-precision policy
(param_dtype=bf16, src/zeroband/train.py:144-146).
"""
from __future__ import annotations

import torch
import torch.nn.functional as F

from . import attention as A
from . import kernels as K


def _bf16(t: torch.Tensor) -> torch.Tensor:
    return t if t.dtype == torch.bfloat16 else t.to(torch.bfloat16)


# ------------------------------------------------------------------------------------------ linear
class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w):
        xb, wb = _bf16(x).contiguous(), _bf16(w).contiguous()
        ctx.save_for_backward(xb, wb)
        ctx.w_dtype = w.dtype
        return K.gemm(xb, wb)

    @staticmethod
    def backward(ctx, dy):
        xb, wb = ctx.saved_tensors
        dy = _bf16(dy).contiguous()
        dx = K.gemm(dy, wb, b_mn=True) if ctx.needs_input_grad[0] else None
        dw = None
        if ctx.needs_input_grad[1]:
            dw = K.gemm(dy, xb, a_mn=True, b_mn=True, out_dtype=torch.float32).to(ctx.w_dtype)
        return dx, dw


def linear(x: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """``x @ w.T`` for 2-D ``x``."""
    if not x.is_cuda:
        return F.linear(x, w.to(x.dtype))
    return _Linear.apply(x, w)


# ------------------------------------------------------------------------------------------ rmsnorm
class _RMSNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps):
        xb, wb = _bf16(x).contiguous(), _bf16(w).contiguous()
        y, rstd = K.rmsnorm_fwd(xb, wb, eps)
        ctx.save_for_backward(xb, wb, rstd)
        ctx.w_dtype = w.dtype
        return y

    @staticmethod
    def backward(ctx, dy):
        xb, wb, rstd = ctx.saved_tensors
        dw = torch.empty(wb.numel(), dtype=torch.float32, device=xb.device)     # overwritten (accumulate_dw=False)
        dx = K.rmsnorm_bwd(xb, wb, rstd, _bf16(dy).contiguous(), dw, accumulate_dw=False)
        return dx, dw.to(ctx.w_dtype), None


def rmsnorm(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    if not x.is_cuda:
        xf = x.float()
        return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()).to(x.dtype)
    shp = x.shape
    return _RMSNorm.apply(x.reshape(-1, shp[-1]), w, eps).reshape(shp)


# ------------------------------------------------------------------------------------------ rope
class _Rope(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, table, seq_len, n_rot, hd):
        ctx.save_for_backward(table)
        ctx.meta = (seq_len, n_rot, hd)
        return K.rope_(_bf16(qkv).contiguous().clone(), table, seq_len, n_rot, hd)

    @staticmethod
    def backward(ctx, d):
        (table,) = ctx.saved_tensors
        seq_len, n_rot, hd = ctx.meta
        return K.rope_(_bf16(d).contiguous().clone(), table, seq_len, n_rot, hd, backward=True), None, None, None, None


def rope(qkv: torch.Tensor, table: torch.Tensor, seq_len: int, n_rot_heads: int, head_dim: int) -> torch.Tensor:
    """Rotate the first ``n_rot_heads`` heads of each row (interleaved pairs); position = row % seq_len."""
    if qkv.is_cuda:
        return _Rope.apply(qkv, table, seq_len, n_rot_heads, head_dim)
    M = qkv.shape[0]
    rot = qkv[:, : n_rot_heads * head_dim].float().reshape(M, n_rot_heads, head_dim // 2, 2)
    cs = table[torch.arange(M, device=qkv.device) % seq_len][:, None].to(rot.dtype)
    re = rot[..., 0] * cs[..., 0] - rot[..., 1] * cs[..., 1]
    im = rot[..., 0] * cs[..., 1] + rot[..., 1] * cs[..., 0]
    out = torch.stack([re, im], -1).reshape(M, -1).to(qkv.dtype)
    return torch.cat([out, qkv[:, n_rot_heads * head_dim:]], -1)


# ------------------------------------------------------------------------------------------ swiglu
class _SwiGLU(torch.autograd.Function):
    @staticmethod
    def forward(ctx, h13):
        hb = _bf16(h13).contiguous()
        ctx.save_for_backward(hb)
        return K.swiglu_fwd(hb)

    @staticmethod
    def backward(ctx, d):
        (hb,) = ctx.saved_tensors
        return K.swiglu_bwd(hb, _bf16(d).contiguous())


def swiglu(h13: torch.Tensor) -> torch.Tensor:
    """``silu(h13[:, :F]) * h13[:, F:]``."""
    if h13.is_cuda:
        return _SwiGLU.apply(h13)
    Fdim = h13.shape[1] // 2
    return F.silu(h13[:, :Fdim]) * h13[:, Fdim:]


# ------------------------------------------------------------------------------------------ attention
class _Attention(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, seq_start, H, KV, hd):
        qb = _bf16(qkv).contiguous()
        o, lse2 = A.attention_fwd(qb, seq_start, H, KV, hd)
        ctx.save_for_backward(qb, o, lse2, seq_start)
        ctx.meta = (H, KV, hd)
        return o

    @staticmethod
    def backward(ctx, do):
        qb, o, lse2, seq_start = ctx.saved_tensors
        H, KV, hd = ctx.meta
        return A.attention_bwd(qb, o, _bf16(do).contiguous(), lse2, seq_start, H, KV, hd), None, None, None, None


def attention(qkv: torch.Tensor, seq_start: torch.Tensor, H: int, KV: int, hd: int) -> torch.Tensor:
    if qkv.is_cuda:
        return _Attention.apply(qkv, seq_start, H, KV, hd)
    return A.attention_reference(qkv, seq_start, H, KV, hd).to(qkv.dtype)


# ------------------------------------------------------------------------------------------ fused blocks
def _stack_bf16(*ws: torch.Tensor) -> torch.Tensor:
    """Weights of equal width below one another in one bf16 matrix."""
    return torch.cat(ws, out=torch.empty(sum(w.shape[0] for w in ws), ws[0].shape[1], dtype=torch.bfloat16, device=ws[0].device))


def _stacked_wgrads(ctx, dy: torch.Tensor, xb: torch.Tensor, first: int, rows) -> list[torch.Tensor | None]:
    """One weight gradient per stacked weight, each from its columns of ``dy`` in place and into a tensor of its own."""
    if all(ctx.needs_input_grad[first + i] for i in range(len(rows))):
        return [dw.to(dt) for dw, dt in zip(K.gemm_row_parts(dy, xb, tuple(rows)), ctx.w_dtypes)]
    out, r = [], 0
    for i, n in enumerate(rows):
        dw = None
        if ctx.needs_input_grad[first + i]:
            dw = K.gemm(dy[:, r: r + n], xb, a_mn=True, b_mn=True, out_dtype=torch.float32).to(ctx.w_dtypes[i])
        out.append(dw)
        r += n
    return out


class _SelfAttention(torch.autograd.Function):
    """q, k and v projections in one GEMM whose epilogue rotates q and k, then attention. As separate linear, cat, rope and
    attention nodes a block took 14 more launches and 5 more copies of activation size."""

    @staticmethod
    def forward(ctx, x, wq, wk, wv, table, seq_start, seq_len, H, KV, hd):
        xb, wb = _bf16(x).contiguous(), _stack_bf16(wq, wk, wv)
        qkv = torch.empty(xb.shape[0], wb.shape[0], dtype=torch.bfloat16, device=xb.device)
        K.gemm_rope(xb, wb, qkv, table, seq_len, H + KV, hd)
        o, lse2 = A.attention_fwd(qkv, seq_start, H, KV, hd)
        ctx.save_for_backward(xb, wb, qkv, o, lse2, table, seq_start)
        ctx.meta = (seq_len, H, KV, hd)
        ctx.w_dtypes = (wq.dtype, wk.dtype, wv.dtype)
        return o

    @staticmethod
    def backward(ctx, do):
        xb, wb, qkv, o, lse2, table, seq_start = ctx.saved_tensors
        seq_len, H, KV, hd = ctx.meta
        dqkv = A.attention_bwd(qkv, o, _bf16(do).contiguous(), lse2, seq_start, H, KV, hd, rope_table=table, seq_len=seq_len)
        dx = K.gemm(dqkv, wb, b_mn=True) if ctx.needs_input_grad[0] else None
        return dx, *_stacked_wgrads(ctx, dqkv, xb, 1, (H * hd, KV * hd, KV * hd)), None, None, None, None, None, None


def self_attention(x, wq, wk, wv, table, seq_start, seq_len: int, H: int, KV: int, hd: int) -> torch.Tensor:
    """``attention(rope(x @ [wq; wk; wv].T))`` for 2-D ``x``: what ``linear``, ``rope`` and ``attention`` compute one by one."""
    if x.is_cuda:
        return _SelfAttention.apply(x, wq, wk, wv, table, seq_start, seq_len, H, KV, hd)
    qkv = torch.cat([linear(x, wq), linear(x, wk), linear(x, wv)], -1)
    return attention(rope(qkv, table, seq_len, H + KV, hd), seq_start, H, KV, hd)


class _SwiGLULinear(torch.autograd.Function):
    """gate and up projections in one GEMM whose epilogue takes the SwiGLU."""

    @staticmethod
    def forward(ctx, x, w1, w3):
        xb, wb = _bf16(x).contiguous(), _stack_bf16(w1, w3)
        h13 = torch.empty(xb.shape[0], wb.shape[0], dtype=torch.bfloat16, device=xb.device)
        act = torch.empty(xb.shape[0], w1.shape[0], dtype=torch.bfloat16, device=xb.device)
        K.gemm_swiglu(xb, wb, h13, act)
        ctx.save_for_backward(xb, wb, h13)
        ctx.w_dtypes = (w1.dtype, w3.dtype)
        return act

    @staticmethod
    def backward(ctx, d):
        xb, wb, h13 = ctx.saved_tensors
        dh13 = K.swiglu_bwd(h13, _bf16(d).contiguous())
        dx = K.gemm(dh13, wb, b_mn=True) if ctx.needs_input_grad[0] else None
        F_ = wb.shape[0] // 2
        return dx, *_stacked_wgrads(ctx, dh13, xb, 1, (F_, F_))


def swiglu_linear(x, w1, w3) -> torch.Tensor:
    """``swiglu(x @ [w1; w3].T)`` for 2-D ``x``."""
    if x.is_cuda:
        return _SwiGLULinear.apply(x, w1, w3)
    return swiglu(torch.cat([linear(x, w1), linear(x, w3)], -1))
