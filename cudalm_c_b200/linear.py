"""Host-side mirror of the reference's GEMM wrappers on quantised weights
(g_ab / g_abt / g_ab_res / g_abt_b / g_atb, cudalm.cu:3133-3202) and the decode GEMV.

`layout` says how the 4-bit codes are stored relative to Y = X W:
KN = codes of W[K,N] (the reference's own [in,out] storage, applied with g_ab),
NK = codes of W[N,K] (applied with g_abt)."""
import torch

from ._lib import BF16, F32, KN, NK, Qkv, calls, check, lib, ptr, stream_ptr  # noqa: F401


def _dt(t):
    if t.dtype == torch.bfloat16:
        return BF16
    if t.dtype == torch.float32:
        return F32
    raise TypeError("activations must be float32 or bfloat16")


def linear_fwd(X, codes, scales, layout, N, R=None, out=None):
    """Y[M,N] = X[M,K] @ deq(W) (+ R)   -- g_ab / g_abt / g_ab_res."""
    M, K = X.shape
    Y = out if out is not None else X.new_empty((M, N))
    calls.linear_fwd(Y, X, codes, scales, layout, M, K, N, R, _dt(X), stream_ptr())
    return Y


def linear_dgrad(dY, codes, scales, layout, K, beta=0.0, out=None):
    """dX[M,K] = beta*dX + dY[M,N] @ deq(W)^T   -- g_abt_b / g_ab."""
    M, N = dY.shape
    dX = out if out is not None else dY.new_empty((M, K))
    calls.linear_dgrad(dX, dY, codes, scales, layout, M, K, N, beta, _dt(dY), stream_ptr())
    return dX


def linear_wgrad(dW, dY, X, layout, beta=1.0):
    """dW (fp32, shape of W) = beta*dW + X^T dY (KN) or dY^T X (NK)   -- g_atb."""
    M, K = X.shape
    N = dY.shape[1]
    calls.linear_wgrad(dW, dY, X, layout, M, K, N, beta, _dt(X), stream_ptr())
    return dW


def _qkv(M, D, KD, ws, cosb, sinb, T):
    a = Qkv(M, D, KD, T)
    for i, (codes, scales) in enumerate(ws):
        a.codes[i], a.scales[i] = ptr(codes), ptr(scales)
    a.cosb, a.sinb = ptr(cosb), ptr(sinb)
    return a


def qkv_fwd(X, ws, KD, cosb, sinb, T):
    """q, k, v = X @ deq(W) for ws = three (codes, scales) pairs [D, D], [D, KD], [D, KD] (layout KN, bf16), q and k rotated."""
    M, D = X.shape
    q, k, v = X.new_empty((M, D)), X.new_empty((M, KD)), X.new_empty((M, KD))
    check(lib().qlmb_qkv_fwd(_qkv(M, D, KD, ws, cosb, sinb, T), ptr(q), ptr(k), ptr(v), ptr(X), stream_ptr()))
    return q, k, v


def qkv_bwd(dWs, dq, dk, dv, X, ws, cosb, sinb, T, beta=1.0):
    """dX of qkv_fwd's projections (dq and dk rotated back already); dWs (fp32) = beta * dWs + X^T [dq | dk | dv]."""
    M, D = X.shape
    dX = torch.empty_like(X)
    check(lib().qlmb_qkv_bwd(_qkv(M, D, dk.shape[1], ws, cosb, sinb, T), ptr(dX), ptr(dWs[0]), ptr(dWs[1]), ptr(dWs[2]), ptr(dq),
                             ptr(dk), ptr(dv), ptr(X), beta, stream_ptr()))
    return dX


def gemv_decode(X, codes, scales, layout, N, out=None):
    """Y[B,N] = X[B,K] @ deq(W) for B <= 64 live decode slots."""
    B, K = X.shape
    Y = out if out is not None else X.new_empty((B, N))
    calls.gemv_decode(Y, X, codes, scales, layout, B, K, N, _dt(X), stream_ptr())
    return Y
