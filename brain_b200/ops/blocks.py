"""A whole transformer block as one autograd node.

Forward and backward issue the launches that the block's operators issue one by one (``functional``, ``attention``), in
their order and with their arguments.  What it saves is the host: an operator is an autograd node with its own Python
frames, 25 us a launch where a kernel of a small model takes 7, so a step on the command line's default model was bound by
it.  The sum of the two gradients of the residual stream goes into the norm's backward kernel.

A block takes this form (``fused_ok``) where its parameters accumulate into ``main_grad`` and nothing sits between its
operators (adapters, tensor parallelism, tuning); else it runs operator by operator."""
from __future__ import annotations

import math
from ctypes import c_long

import torch

from ..utils import tune as _tune
from . import functional as F
from ._cuda import call, stream_ptr


def fused_ok(x, params) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and _tune._TUNER is None and x.numel() > 0
            and all(p.requires_grad and p.dtype == torch.bfloat16 and getattr(p, "main_grad", None) is not None for p in params))


def _project(x, w, bias, n, s):
    """x [n, k] @ w [m, k]^T (+ bias)"""
    m, k = w.shape
    assert x.shape == (n, k) and w.stride(1) == 1, (x.shape, w.shape, w.stride())
    y = torch.empty(n, m, device=x.device, dtype=torch.bfloat16)
    call("gemm_bf16", x, w, y, bias, n, m, k, k, w.stride(0), m, 0, 0, 0, 1.0, 0, 0, s)
    return y


def _project_back(dy, x, w, wp, bp, n, s):
    """Gradient of _project: adds into the parameters' main_grad, returns dx."""
    m, k = w.shape
    mg = wp.main_grad
    assert dy.shape == (n, m) and x.shape == (n, k), (dy.shape, x.shape, w.shape)
    assert mg.shape == w.shape and mg.stride(1) == 1 and mg.dtype == torch.float32, (mg.shape, mg.stride(), mg.dtype)
    dx = torch.empty(n, k, device=dy.device, dtype=torch.bfloat16)
    call("gemm_bf16", dy, w, dx, None, n, k, m, m, w.stride(0), k, 0, 1, 0, 1.0, 0, 0, s)
    call("gemm_bf16", dy, x, mg, None, m, k, n, m, k, mg.stride(0), 1, 1, 2, 1.0, 0, 0, s)
    F._notify(wp)
    if bp is not None:
        call("colsum", dy, None, None, None, bp.main_grad, n, m, m, 0, s)
        F._notify(bp)
    return dx


class _QwenBlock(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, cos, sin, pos, dims, *params):
        ln1, wqkv, bqkv, q_norm, k_norm, wo, ln2, gate_up, down = params
        B, T, hq, hk, hd, eps = dims
        x = x.contiguous()
        n, d = x.shape
        s, new, f32 = stream_ptr(), x.new_empty, torch.float32
        h, rstd1 = new(n, d), new(n, dtype=f32)
        x1 = x
        if delta is None:
            call("rmsnorm_fwd", x, None, ln1, h, None, rstd1, n, d, eps, s)
        else:
            x1 = new(n, d)
            call("rmsnorm_fwd", delta.contiguous(), x, ln1, h, x1, rstd1, n, d, eps, s)
        qkv = _project(h, wqkv, bqkv.float() if bqkv is not None else None, n, s)
        qw, qkw, ld = hq * hd, (hq + hk) * hd, (hq + 2 * hk) * hd
        qk, rstd = new(n, qkw), new(n * (hq + hk), dtype=f32) if q_norm is not None else None
        call("qknorm_rope_fwd", qkv, ld, q_norm, k_norm, cos, sin, pos, qk, qkw, rstd, n, hq, hk, hd, eps, s)
        out, lse = new(n, qw), new(B, hq, T, dtype=f32)
        call("flash_fwd", qk, qkw, qk[:, qw:], qkw, qkv[:, qkw:], ld, out, qw, lse, B, T, T, hq, hk, hd, 1.0 / math.sqrt(hd), 1, s)
        a = _project(out, wo, None, n, s)
        h2, x2, rstd2 = new(n, d), new(n, d), new(n, dtype=f32)
        call("rmsnorm_fwd", a, x1, ln2, h2, x2, rstd2, n, d, eps, s)
        gu = _project(h2, gate_up, None, n, s)
        ff = gu.shape[1] // 2
        act = new(n, ff)
        call("swiglu_fwd", gu, act, c_long(n), ff, s)
        y = _project(act, down, None, n, s)
        ctx.save_for_backward(x1, h, rstd1, qkv, qk, rstd, out, lse, x2, h2, rstd2, gu, act, cos, sin, pos, ln1, wqkv, q_norm, k_norm, wo,
                              ln2, gate_up, down)
        ctx.params, ctx.dims, ctx.has_delta = params, dims, delta is not None
        return x2, y

    @staticmethod
    def backward(ctx, dx2, dy):
        (x1, h, rstd1, qkv, qk, rstd, out, lse, x2, h2, rstd2, gu, act, cos, sin, pos, ln1, wqkv, q_norm, k_norm, wo, ln2, gate_up,
         down) = ctx.saved_tensors
        p_ln1, p_wqkv, p_bqkv, p_qn, p_kn, p_wo, p_ln2, p_gu, p_down = ctx.params
        B, T, hq, hk, hd, eps = ctx.dims
        n, d = x1.shape
        s, new = stream_ptr(), x1.new_empty
        dx2, dy = dx2.contiguous(), dy.contiguous()
        dact = _project_back(dy, act, down, p_down, None, n, s)
        dgu = torch.empty_like(gu)
        call("swiglu_bwd", dact, gu, dgu, c_long(n), act.shape[1], s)
        dh = _project_back(dgu, h2, gate_up, p_gu, None, n, s)
        dx1 = new(n, d)
        call("rmsnorm_bwd", dh, x2, ln2, rstd2, dx2, dx1, p_ln2.main_grad, n, d, s)
        F._notify(p_ln2)
        dout = _project_back(dx1, out, wo, p_wo, None, n, s)
        qw, qkw, ld = hq * hd, (hq + hk) * hd, (hq + 2 * hk) * hd
        dqkv, dqk, row_dot = torch.empty_like(qkv), torch.empty_like(qk), torch.empty_like(lse)
        call("flash_bwd", qk, qkw, qk[:, qw:], qkw, qkv[:, qkw:], ld, out, qw, dout, qw, lse, row_dot, dqk, qkw, dqk[:, qw:], qkw,
             dqkv[:, qkw:], ld, B, T, T, hq, hk, hd, 1.0 / math.sqrt(hd), 1, s)
        normed = q_norm is not None
        call("qknorm_rope_bwd", dqk, qkw, qkv, ld, q_norm, k_norm, rstd, cos, sin, pos, dqkv, ld, p_qn.main_grad if normed else None,
             p_kn.main_grad if normed else None, n, hq, hk, hd, s)
        if normed:
            F._notify(p_qn)
            F._notify(p_kn)
        dh = _project_back(dqkv, h, wqkv, p_wqkv, p_bqkv, n, s)
        dx = new(n, d)
        call("rmsnorm_bwd", dh, x1, ln1, rstd1, dx1, dx, p_ln1.main_grad, n, d, s)
        F._notify(p_ln1)
        return (dx, dx if ctx.has_delta else None) + (None,) * 13


def qwen_block(x, delta, cos, sin, pos, dims, params):
    """(residual stream, unadded feed-forward output) of a pre-norm block with QK-norm, rotation and SwiGLU; ``dims``:
    B, T, query heads, key / value heads, head size, eps; ``params``: ln1, wqkv, bqkv or None, q_norm, k_norm (or None),
    wo, ln2, gate_up, down."""
    return _QwenBlock.apply(x, delta, cos, sin, pos, dims, *params)


class _GptBlock(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, delta, dims, *params):
        ln1_w, ln1_b, qkv_w, qkv_b, out_w, out_b, ln2_w, ln2_b, fc_w, fc_b, proj_w, proj_b = params
        B, T, H, eps = dims
        x = x.contiguous()
        n, d = x.shape
        hd = d // H
        s, new, f32 = stream_ptr(), x.new_empty, torch.float32
        h, mean1, rstd1 = new(n, d), new(n, dtype=f32), new(n, dtype=f32)
        x1 = x if delta is None else new(n, d)
        call("layernorm_res_fwd", x if delta is None else delta.contiguous(), None if delta is None else x, ln1_w, ln1_b, h,
             None if delta is None else x1, mean1, rstd1, n, d, eps, s)
        qkv = _project(h, qkv_w, qkv_b.float(), n, s)
        ld = 3 * d
        out, lse = new(n, d), new(B, H, T, dtype=f32)
        call("flash_fwd", qkv, ld, qkv[:, d:], ld, qkv[:, 2 * d:], ld, out, d, lse, B, T, T, H, H, hd, 1.0 / math.sqrt(hd), 1, s)
        a = _project(out, out_w, out_b.float(), n, s)
        h2, x2, mean2, rstd2 = new(n, d), new(n, d), new(n, dtype=f32), new(n, dtype=f32)
        call("layernorm_res_fwd", a, x1, ln2_w, ln2_b, h2, x2, mean2, rstd2, n, d, eps, s)
        u = _project(h2, fc_w, fc_b.float(), n, s)
        act = torch.empty_like(u)
        call("gelu_fwd", u, act, c_long(u.numel()), s)
        y = _project(act, proj_w, proj_b.float(), n, s)
        ctx.save_for_backward(x1, h, mean1, rstd1, qkv, out, lse, x2, h2, mean2, rstd2, u, act, ln1_w, qkv_w, out_w, ln2_w, fc_w, proj_w)
        ctx.params, ctx.dims, ctx.has_delta = params, dims, delta is not None
        return x2, y

    @staticmethod
    def backward(ctx, dx2, dy):
        x1, h, mean1, rstd1, qkv, out, lse, x2, h2, mean2, rstd2, u, act, ln1_w, qkv_w, out_w, ln2_w, fc_w, proj_w = ctx.saved_tensors
        p_ln1w, p_ln1b, p_qkvw, p_qkvb, p_outw, p_outb, p_ln2w, p_ln2b, p_fcw, p_fcb, p_projw, p_projb = ctx.params
        B, T, H, eps = ctx.dims
        n, d = x1.shape
        hd, ld = d // H, 3 * d
        s = stream_ptr()
        dx2, dy = dx2.contiguous(), dy.contiguous()

        def norm_back(dh, xin, g, mean, rstd, dres, pw, pb):
            dx = torch.empty_like(xin)
            call("layernorm_bwd", dh, xin, g, mean, rstd, dres, dx, pw.main_grad, pb.main_grad, n, d, s)
            F._notify(pw)
            F._notify(pb)
            return dx

        dact = _project_back(dy, act, proj_w, p_projw, p_projb, n, s)
        du = torch.empty_like(u)
        call("gelu_bwd", dact, u, du, c_long(u.numel()), s)
        dh = _project_back(du, h2, fc_w, p_fcw, p_fcb, n, s)
        dx1 = norm_back(dh, x2, ln2_w, mean2, rstd2, dx2, p_ln2w, p_ln2b)
        dout = _project_back(dx1, out, out_w, p_outw, p_outb, n, s)
        dqkv, row_dot = torch.empty_like(qkv), torch.empty_like(lse)
        call("flash_bwd", qkv, ld, qkv[:, d:], ld, qkv[:, 2 * d:], ld, out, d, dout, d, lse, row_dot, dqkv, ld, dqkv[:, d:], ld,
             dqkv[:, 2 * d:], ld, B, T, T, H, H, hd, 1.0 / math.sqrt(hd), 1, s)
        dh = _project_back(dqkv, h, qkv_w, p_qkvw, p_qkvb, n, s)
        dx = norm_back(dh, x1, ln1_w, mean1, rstd1, dx1, p_ln1w, p_ln1b)
        return (dx, dx if ctx.has_delta else None) + (None,) * 13


def gpt_block(x, delta, dims, params):
    """(residual stream, unadded feed-forward output) of a pre-LayerNorm block with biases and tanh-GELU; ``dims``: B, T,
    heads, eps; ``params``: weight and bias of ln1, qkv, out, ln2, fc, proj."""
    return _GptBlock.apply(x, delta, dims, *params)
