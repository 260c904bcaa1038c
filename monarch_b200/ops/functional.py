"""Tensor-level entry points of the hand-written sm_100a kernels.

Every function dispatches on the device of its inputs: CUDA tensors go to the kernel
library (and fail loudly if it is missing), CPU tensors go to the fp32 PyTorch
reference so that engines and tests run without a GPU.
"""
from __future__ import annotations

import os

import torch

from . import kernels as K
from . import reference as R

bf16 = torch.bfloat16


def _p(t):
    return 0 if t is None else t.data_ptr()


def _rowmajor(t: torch.Tensor):
    """(t with unit inner stride, its leading dimension)."""
    assert t.dim() == 2
    ld, inner = t.stride()
    if inner != 1 or ld < t.shape[1]:
        t = t.contiguous()
        ld = t.stride(0)
    return t, ld


def gemm(a, b, *, a_mn=False, b_mn=False, out=None, residual=None, accumulate=False):
    """out[M,N] = opA(a) @ opB(b) (+ residual) (+ out when ``accumulate``).

    ``a`` is [M,K] (``a_mn=False``) or [K,M] (``a_mn=True``); ``b`` is [N,K]
    (``b_mn=False``, i.e. out = a @ b.T) or [K,N] (``b_mn=True``).  bf16 in, fp32
    accumulation on the tensor cores (tcgen05, accumulator in TMEM), bf16 out.
    """
    a, lda = _rowmajor(a)
    b, ldb = _rowmajor(b)
    M, Ka = a.shape
    if a_mn:
        M, Ka = Ka, M
    N, Kb = b.shape
    if b_mn:
        N, Kb = Kb, N
    assert Ka == Kb, (a.shape, b.shape, a_mn, b_mn)
    if out is None:
        assert not accumulate
        out = torch.empty(M, N, dtype=a.dtype, device=a.device)
        ldc = N
    else:
        ldc, inner = out.stride()
        assert out.shape == (M, N) and inner == 1
    if not a.is_cuda:
        out.copy_(R.gemm(a, b, a_mn, b_mn, residual, out if accumulate else None).to(out.dtype))
        return out
    assert a.dtype == bf16 and b.dtype == bf16 and out.dtype == bf16
    res, ldr = 0, 0
    if residual is not None:
        ldr, inner = residual.stride()
        assert residual.shape == (M, N) and inner == 1 and residual.dtype == bf16
        res = residual.data_ptr()
    rc = K.lib().mb200_gemm_bf16(
        a.data_ptr(), b.data_ptr(), out.data_ptr(), res, M, N, Ka, lda, ldb, ldc, ldr,
        int(a_mn), int(b_mn), int(accumulate), K.status_ptr(a), K.stream_ptr())
    K.check(rc, "gemm_bf16")
    return out


def rmsnorm_fwd(x, w, eps=1e-5):
    rows, d = x.shape
    if not x.is_cuda:
        y, rstd = R.rmsnorm_fwd(x, w, eps)
        return y.to(x.dtype), rstd
    x = x.contiguous()
    y = torch.empty_like(x)
    rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
    K.check(K.lib().mb200_rmsnorm_fwd(x.data_ptr(), w.data_ptr(), y.data_ptr(), rstd.data_ptr(),
                                      rows, d, eps, K.stream_ptr()), "rmsnorm_fwd")
    return y, rstd


_rms_most_blocks: dict = {}   # device index -> mb200_rmsnorm_bwd_blocks of many rows


def rmsnorm_bwd(dy, x, w, rstd, dw_out, accumulate=False, dres=None):
    """Returns dx (+ ``dres``); writes (or adds) the weight gradient into ``dw_out``."""
    rows, d = x.shape
    if not x.is_cuda:
        dx, dw = R.rmsnorm_bwd(dy, x, w, rstd)
        if dres is not None:
            dx = dx + dres.float()
        if accumulate:
            dw = dw + dw_out.float()
        dw_out.copy_(dw.to(dw_out.dtype))
        return dx.to(x.dtype)
    dy = dy.contiguous()
    dx = torch.empty_like(x)
    dev = x.get_device()
    most = _rms_most_blocks.get(dev)
    if most is None:
        most = _rms_most_blocks[dev] = K.lib().mb200_rmsnorm_bwd_blocks(1 << 30)
    # of this call alone: another stream's call may run between the two kernels that use it
    part = torch.empty((rows if rows < most else most) * d, dtype=torch.float32, device=x.device)
    K.check(K.lib().mb200_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(),
                                      _p(dres), dx.data_ptr(), part.data_ptr(), dw_out.data_ptr(),
                                      int(accumulate), rows, d, K.status_ptr(x), K.stream_ptr()),
            "rmsnorm_bwd", 2)
    return dx


def rope_(qkv, cos, sin, seq_len, n_rot_heads, hd, inverse=False):
    """In-place rotary embedding on the first ``n_rot_heads`` heads of each row."""
    rows = qkv.shape[0]
    if not qkv.is_cuda:
        x = qkv[:, : n_rot_heads * hd].float().reshape(rows, n_rot_heads, hd)
        y = R.rope(x, cos, sin, seq_len, inverse)
        qkv[:, : n_rot_heads * hd] = y.reshape(rows, -1).to(qkv.dtype)
        return qkv
    assert qkv.stride(1) == 1
    K.check(K.lib().mb200_rope_inplace(qkv.data_ptr(), cos.data_ptr(), sin.data_ptr(), rows,
                                       seq_len, n_rot_heads, hd, qkv.stride(0), int(inverse),
                                       K.stream_ptr()), "rope")
    return qkv


def swiglu_fwd(gu, out=None):
    rows, F2 = gu.shape
    if not gu.is_cuda:
        h = R.swiglu_fwd(gu).to(gu.dtype)
        return h if out is None else out.copy_(h)
    h = torch.empty(rows, F2 // 2, dtype=gu.dtype, device=gu.device) if out is None else out
    K.check(K.lib().mb200_swiglu_fwd(gu.data_ptr(), h.data_ptr(), rows, F2 // 2, K.stream_ptr()),
            "swiglu_fwd")
    return h


def swiglu_bwd(gu, dh, out=None):
    rows, F2 = gu.shape
    if not gu.is_cuda:
        r = R.swiglu_bwd(gu, dh).to(gu.dtype)
        if out is not None:
            out.copy_(r)
            return out
        return r
    dgu = torch.empty_like(gu) if out is None else out
    K.check(K.lib().mb200_swiglu_bwd(gu.data_ptr(), dh.data_ptr(), dgu.data_ptr(), rows, F2 // 2,
                                     K.stream_ptr()), "swiglu_bwd")
    return dgu


_NOT_FUSED, _TWO_KERNELS = 1003, 1004   # MB200_NOT_FUSED, MB200_TWO_KERNELS
# Rows x F for which the library most likely launches two kernels: more than one wave of small
# tiles and less than pair tiles fuse for.  The matrix between the two is ready then; elsewhere
# the library asks for it, a call of 2 us more.
_LIKELY_TWO = (1 << 20, 1 << 23)


def gemm_swiglu(a, w_gu, keep_gu=True):
    """``gu = a @ w_gu.T`` ([rows, 2F]) and ``h = swiglu_fwd(gu)``; returns (h, gu), without
    ``keep_gu`` (h, None).  One kernel where that is faster, with the bits of the two."""
    T, F = a.shape[0], w_gu.shape[0] // 2
    if a.is_cuda and T and not F % 64 and a.dtype == bf16 and w_gu.dtype == bf16:
        a, lda = _rowmajor(a)
        w_gu, ldw = _rowmajor(w_gu)
        Kd = a.shape[1]
        assert w_gu.shape == (2 * F, Kd), (a.shape, w_gu.shape)
        h = torch.empty(T, F, dtype=bf16, device=a.device)
        gu = None
        if keep_gu or _LIKELY_TWO[0] <= T * F <= _LIKELY_TWO[1]:
            gu = torch.empty(T, 2 * F, dtype=bf16, device=a.device)

        def run(gu):
            return K.lib().mb200_gemm_swiglu_fwd(
                a.data_ptr(), w_gu.data_ptr(), h.data_ptr(), _p(gu), T, F, Kd, lda, ldw, F, 2 * F,
                int(keep_gu), K.status_ptr(a), K.stream_ptr())

        rc = run(gu)
        if rc == _NOT_FUSED:
            gu = torch.empty(T, 2 * F, dtype=bf16, device=a.device)
            rc = run(gu)
        if rc == _TWO_KERNELS:
            K.check(0, "gemm_swiglu_fwd", 2)
        else:
            K.check(rc, "gemm_swiglu_fwd")
        return h, (gu if keep_gu else None)
    gu = gemm(a, w_gu)
    return swiglu_fwd(gu), (gu if keep_gu else None)


def gemm_swiglu_bwd(dy, w_down, gu):
    """``swiglu_bwd(gu, dy @ w_down)``; one kernel where that is faster, with the bits of the
    two."""
    T, F = dy.shape[0], w_down.shape[1]
    if (dy.is_cuda and T and not F % 32 and dy.dtype == bf16 and w_down.dtype == bf16
            and gu.dtype == bf16 and gu.is_contiguous() and not gu.data_ptr() & 15):
        dy, lda = _rowmajor(dy)
        w_down, ldw = _rowmajor(w_down)
        Kd = dy.shape[1]
        assert w_down.shape[0] == Kd and gu.shape == (T, 2 * F), (dy.shape, w_down.shape, gu.shape)
        dgu = torch.empty_like(gu)
        dh = None
        if _LIKELY_TWO[0] <= T * F <= _LIKELY_TWO[1]:
            dh = torch.empty(T, F, dtype=bf16, device=dy.device)

        def run(dh):
            return K.lib().mb200_gemm_swiglu_bwd(
                dy.data_ptr(), w_down.data_ptr(), gu.data_ptr(), dgu.data_ptr(), _p(dh), T, F, Kd,
                lda, ldw, 2 * F, K.status_ptr(dy), K.stream_ptr())

        rc = run(dh)
        if rc == _NOT_FUSED:
            dh = torch.empty(T, F, dtype=bf16, device=dy.device)
            rc = run(dh)
        if rc == _TWO_KERNELS:
            K.check(0, "gemm_swiglu_bwd", 2)
        else:
            K.check(rc, "gemm_swiglu_bwd")
        return dgu
    return swiglu_bwd(gu, gemm(dy, w_down, b_mn=True))


def cross_entropy_(logits, targets, grad_scale):
    """Per-row loss; ``logits`` is overwritten with d(loss_sum * grad_scale)/d(logits)."""
    rows, V = logits.shape
    if not logits.is_cuda:
        loss, g = R.cross_entropy(logits, targets, grad_scale)
        logits.copy_(g.to(logits.dtype))
        return loss
    loss = torch.empty(rows, dtype=torch.float32, device=logits.device)
    assert targets.dtype == torch.int64 and logits.stride(1) == 1
    K.check(K.lib().mb200_cross_entropy_fwd_bwd(logits.data_ptr(), targets.data_ptr(),
                                                loss.data_ptr(), rows, V, logits.stride(0),
                                                grad_scale, K.stream_ptr()), "cross_entropy")
    return loss


def adamw_(p, m, v, g, p_bf16, *, lr, beta1=0.9, beta2=0.95, eps=1e-8, wd=0.1, step=1,
           grad_scale=1.0):
    """Fused AdamW step on flat fp32 master/moment buffers; refreshes the bf16 copy."""
    if not p.is_cuda:
        np_, nm, nv = R.adamw(p, m, v, g, lr, beta1, beta2, eps, wd, step, grad_scale)
        p.copy_(np_)
        m.copy_(nm)
        v.copy_(nv)
        if p_bf16 is not None:
            p_bf16.copy_(p.to(p_bf16.dtype))
        return
    assert p.dtype == torch.float32 and p.is_contiguous() and g.is_contiguous()
    K.check(K.lib().mb200_adamw(p.data_ptr(), m.data_ptr(), v.data_ptr(), g.data_ptr(),
                                _p(p_bf16), p.numel(), int(g.dtype == bf16), lr, beta1, beta2, eps,
                                wd, step, grad_scale, K.stream_ptr()), "adamw")


def embedding_fwd(table, ids):
    rows, d = ids.numel(), table.shape[1]
    if not table.is_cuda:
        return table[ids.reshape(-1)]
    out = torch.empty(rows, d, dtype=table.dtype, device=table.device)
    K.check(K.lib().mb200_embedding_fwd(table.data_ptr(), ids.data_ptr(), out.data_ptr(), rows, d,
                                        K.stream_ptr()), "embedding_fwd")
    return out


def embedding_bwd_(dout, ids, dtable):
    """dtable[ids[r]] += dout[r] (atomic)."""
    rows, d = dout.shape
    if not dout.is_cuda:
        dtable.index_add_(0, ids.reshape(-1), dout.to(dtable.dtype))
        return
    K.check(K.lib().mb200_embedding_bwd(dout.data_ptr(), ids.data_ptr(), dtable.data_ptr(), rows,
                                        d, K.stream_ptr()), "embedding_bwd")


def sumsq(x, out=None):
    if out is None:
        out = torch.zeros(1, dtype=torch.float32, device=x.device)
    if not x.is_cuda:
        out += x.float().pow(2).sum()
        return out
    K.check(K.lib().mb200_sumsq(x.data_ptr(), x.numel(), int(x.dtype == bf16), out.data_ptr(),
                                K.stream_ptr()), "sumsq")
    return out


def have_attention_kernel() -> bool:
    """True when the tcgen05 flash-attention kernels (forward and backward) are in the
    loaded library and not disabled with ``MB200_ATTN=sdpa``."""
    if os.environ.get("MB200_ATTN", "") == "sdpa" or not torch.cuda.is_available():
        return False
    return _lib_has_attention()


def _lib_has_attention() -> bool:
    l = K.lib()
    return hasattr(l, "mb200_attn_fwd") and hasattr(l, "mb200_attn_bwd")


class AttnCtx:
    """What attention_bwd needs from attention_fwd."""
    __slots__ = ("qkv", "o", "lse", "B", "S", "Hq", "Hkv", "hd", "scale", "graph")


def attention_fwd(qkv, B, S, Hq, Hkv, hd, scale=None, need_bwd=True):
    """Causal GQA attention on a fused post-RoPE qkv buffer [B*S, (Hq+2Hkv)*hd].

    Returns (o [B*S, Hq*hd], ctx).  On sm_100a the hand-written tcgen05 flash kernel is
    used when the library exports it; otherwise (CPU, or library built without it) the
    math is done by torch SDPA.
    """
    scale = scale if scale is not None else hd ** -0.5
    ctx = AttnCtx()
    ctx.qkv, ctx.B, ctx.S, ctx.Hq, ctx.Hkv, ctx.hd, ctx.scale = qkv, B, S, Hq, Hkv, hd, scale
    ctx.graph = None
    T = B * S
    if qkv.is_cuda and os.environ.get("MB200_ATTN", "") != "sdpa" and _lib_has_attention():
        o = torch.empty(T, Hq * hd, dtype=qkv.dtype, device=qkv.device)
        lse = torch.empty(B, Hq, S, dtype=torch.float32, device=qkv.device)
        q = qkv
        k = qkv[:, Hq * hd:]
        v = qkv[:, (Hq + Hkv) * hd:]
        K.check(K.lib().mb200_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                                       lse.data_ptr(), B, S, Hq, Hkv, hd, qkv.stride(0),
                                       o.stride(0), scale, K.status_ptr(qkv),
                                       K.stream_ptr()), "attn_fwd")
        ctx.o, ctx.lse = o, lse
        return o, ctx
    q = qkv[:, : Hq * hd].reshape(B, S, Hq, hd).transpose(1, 2)
    k = qkv[:, Hq * hd: (Hq + Hkv) * hd].reshape(B, S, Hkv, hd).transpose(1, 2)
    v = qkv[:, (Hq + Hkv) * hd:].reshape(B, S, Hkv, hd).transpose(1, 2)
    if need_bwd:
        q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
    with torch.enable_grad() if need_bwd else torch.no_grad():
        o = torch.nn.functional.scaled_dot_product_attention(q, k, v, is_causal=True, scale=scale,
                                                             enable_gqa=True)
        o2 = o.transpose(1, 2).reshape(T, Hq * hd)
    if need_bwd:
        ctx.graph = (q, k, v, o2)
    ctx.o, ctx.lse = o2.detach(), None
    return ctx.o, ctx


def attention_ctx_from_saved(qkv, saved, B, S, Hq, Hkv, hd, scale=None):
    """Rebuild the backward context from a recomputed qkv and the (o, lse) that the first
    forward kept, without running the attention kernel again."""
    ctx = AttnCtx()
    ctx.qkv, ctx.B, ctx.S, ctx.Hq, ctx.Hkv, ctx.hd = qkv, B, S, Hq, Hkv, hd
    ctx.scale = scale if scale is not None else hd ** -0.5
    ctx.graph = None
    ctx.o, ctx.lse = saved
    return ctx.o, ctx


def attention_bwd(ctx: AttnCtx, do):
    """Gradient w.r.t. the fused (post-RoPE) qkv buffer: [B*S, (Hq+2Hkv)*hd]."""
    B, S, Hq, Hkv, hd = ctx.B, ctx.S, ctx.Hq, ctx.Hkv, ctx.hd
    T = B * S
    dqkv = torch.empty_like(ctx.qkv)
    if ctx.graph is None and ctx.lse is not None:
        qkv = ctx.qkv
        delta = torch.empty(B, Hq, S, dtype=torch.float32, device=qkv.device)
        k = qkv[:, Hq * hd:]
        v = qkv[:, (Hq + Hkv) * hd:]
        dk = dqkv[:, Hq * hd:]
        dv = dqkv[:, (Hq + Hkv) * hd:]
        K.check(K.lib().mb200_attn_bwd(qkv.data_ptr(), k.data_ptr(), v.data_ptr(),
                                       ctx.o.data_ptr(), do.data_ptr(), ctx.lse.data_ptr(),
                                       delta.data_ptr(), dqkv.data_ptr(), dk.data_ptr(),
                                       dv.data_ptr(), B, S, Hq, Hkv, hd, qkv.stride(0),
                                       ctx.o.stride(0), dqkv.stride(0), ctx.scale,
                                       K.status_ptr(qkv), K.stream_ptr()),
                "attn_bwd", 3)
        return dqkv
    q, k, v, o2 = ctx.graph
    dq, dk, dv = torch.autograd.grad(o2, (q, k, v), do)
    dqkv[:, : Hq * hd] = dq.transpose(1, 2).reshape(T, Hq * hd)
    dqkv[:, Hq * hd: (Hq + Hkv) * hd] = dk.transpose(1, 2).reshape(T, Hkv * hd)
    dqkv[:, (Hq + Hkv) * hd:] = dv.transpose(1, 2).reshape(T, Hkv * hd)
    ctx.graph = None
    return dqkv
