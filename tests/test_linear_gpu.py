"""Dequant-fused linears (tcgen05) through the C ABI.
Tolerance (stated by the task): <= 1e-2 relative for bf16 tensor-core operands
against fp32 results, measured both as ||a-b||_F/||b||_F and max|a-b|/max|b|."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import golden

pytestmark = pytest.mark.gpu
TOL = 1e-2
f32 = np.float32


def dev(a, cuda):
    return torch.from_numpy(np.ascontiguousarray(a)).to(cuda)


def rel(a, b):
    a, b = a.float(), b.float()
    return max(float((a - b).norm() / b.norm()), float((a - b).abs().max() / b.abs().max()))


def test_engine_plain_bf16(cuda):
    """TMA + tcgen05 + TMEM pipeline without the dequant warps vs fp32 matmul."""
    import cudalm_c_b200 as q
    from cudalm_c_b200._lib import ptr, stream_ptr
    L = q.lib()
    L.qlmb_selftest_gemm_bf16.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3 + [C.c_void_p]
    torch.manual_seed(1)
    for M, K, N in ((128, 64, 256), (1000, 512, 512), (4096, 1024, 1024)):
        A = torch.randn(M, K, device=cuda).bfloat16(); B = torch.randn(N, K, device=cuda).bfloat16()
        Cc = torch.zeros(M, N, device=cuda)
        q.check(L.qlmb_selftest_gemm_bf16(ptr(Cc), ptr(A), ptr(B), M, K, N, stream_ptr()))
        assert rel(Cc, A.float() @ B.float().T) < 1e-5
    q.check(L.qlmb_check_device(None))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_linear_matches_reference_vectors(cuda, dtype):
    """g_ab / g_abt / g_atb of the reference on its rendered weights (fixture)."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    g = golden("linear")
    X, dY = dev(g["X"], cuda).to(dtype), dev(g["dY"], cuda).to(dtype)
    d, s = dev(g["d"], cuda), dev(g["s"], cuda)
    M, K = X.shape
    N = dY.shape[1]
    for lay, tag in ((KN, "kn"), (NK, "nk")):
        assert rel(linear.linear_fwd(X, d, s, lay, N), dev(g["Y_" + tag], cuda)) < TOL
        assert rel(linear.linear_dgrad(dY, d, s, lay, K), dev(g["dX_" + tag], cuda)) < TOL
        shape = (K, N) if lay == KN else (N, K)
        dW = torch.zeros(shape, device=cuda)
        linear.linear_wgrad(dW, dY, X, lay, beta=1.0)
        assert rel(dW, dev(g["dW_" + tag], cuda)) < TOL


def quantise(cuda, rows, cols, seed):
    from cudalm_c_b200 import qlm
    n = rows * cols
    Q = qlm.Qlm([(0, n)], n, cuda)
    gen = torch.Generator(device=cuda); gen.manual_seed(seed)
    P = torch.randn(n, device=cuda, generator=gen) * 0.02
    Q.init_from(P)                       # P now holds the rendered view s*d
    return Q, P.view(rows, cols)


@pytest.mark.parametrize("layout_name", ["KN", "NK"])
def test_config1_shape(cuda, oracle, layout_name):
    """X[8192,512], W[2048,512] (NK) resp. [512,2048] (KN),
    fwd + dgrad + wgrad with fp32 I/O; full result vs fp32 matmul on the rendered
    view, 32 rows vs the oracle, plus linearity and run-to-run determinism."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    lay = KN if layout_name == "KN" else NK
    M, K, N = 8192, 512, 2048
    Q, W = quantise(cuda, K, N, 3) if lay == KN else quantise(cuda, N, K, 3)
    Wm = W if lay == KN else W.T
    gen = torch.Generator(device=cuda); gen.manual_seed(4)
    X = torch.randn(M, K, device=cuda, generator=gen); dY = torch.randn(M, N, device=cuda, generator=gen)
    Y = linear.linear_fwd(X, Q.d, Q.s, lay, N)
    assert rel(Y, X @ Wm) < TOL
    dX = linear.linear_dgrad(dY, Q.d, Q.s, lay, K)
    assert rel(dX, dY @ Wm.T) < TOL
    dW = torch.zeros_like(W)
    linear.linear_wgrad(dW, dY, X, lay, beta=0.0)
    assert rel(dW, X.T @ dY if lay == KN else dY.T @ X) < TOL
    # oracle on a slice of rows
    dn, sn = Q.d.cpu().numpy(), Q.s.cpu().numpy()
    Yo = oracle.linear_fwd(X[:32].cpu().numpy(), dn, sn, lay, N)
    assert rel(Y[:32], dev(Yo, cuda)) < TOL
    dXo = oracle.linear_dgrad(dY[:32].cpu().numpy(), dn, sn, lay, K)
    assert rel(dX[:32], dev(dXo, cuda)) < TOL
    # size-independent properties: determinism, and linearity in the bf16-exact factor 2
    assert torch.equal(Y, linear.linear_fwd(X, Q.d, Q.s, lay, N))
    assert torch.equal(linear.linear_fwd(2 * X, Q.d, Q.s, lay, N), 2 * Y)
    # residual epilogue and accumulate modes
    R = torch.randn(M, N, device=cuda, generator=gen)
    assert rel(linear.linear_fwd(X, Q.d, Q.s, lay, N, R=R) - R, Y) < 1e-5
    acc = dX.clone()
    linear.linear_dgrad(dY, Q.d, Q.s, lay, K, beta=1.0, out=acc)
    assert rel(acc, 2 * dX) < 1e-6
    dW2 = dW.clone()
    linear.linear_wgrad(dW2, dY, X, lay, beta=1.0)
    assert rel(dW2, 2 * dW) < 1e-6


@pytest.mark.parametrize("M", [1, 127, 129, 300])
def test_ragged_row_counts(cuda, M):
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    K, N = 256, 384
    for lay in (KN, NK):
        Q, W = quantise(cuda, K, N, 7) if lay == KN else quantise(cuda, N, K, 7)
        Wm = W if lay == KN else W.T
        X = torch.randn(M, K, device=cuda).bfloat16(); dY = torch.randn(M, N, device=cuda).bfloat16()
        guard = torch.full((M + 1, N), 7.0, device=cuda, dtype=torch.bfloat16)
        linear.linear_fwd(X, Q.d, Q.s, lay, N, out=guard[:M])
        assert rel(guard[:M], X.float() @ Wm) < TOL
        assert (guard[M] == 7.0).all()            # rows past M are never written
        assert rel(linear.linear_dgrad(dY, Q.d, Q.s, lay, K), dY.float() @ Wm.T) < TOL
        dW = torch.zeros_like(W)
        linear.linear_wgrad(dW, dY, X, lay, beta=0.0)
        assert rel(dW, X.float().T @ dY.float() if lay == KN else dY.float().T @ X.float()) < TOL


def test_empty_and_unsupported(cuda):
    import cudalm_c_b200 as q
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN
    Q, W = quantise(cuda, 128, 128, 9)
    assert linear.linear_fwd(torch.zeros(0, 128, device=cuda), Q.d, Q.s, KN, 128).shape == (0, 128)
    dW = torch.ones(128, 128, device=cuda)
    linear.linear_wgrad(dW, torch.zeros(0, 128, device=cuda), torch.zeros(0, 128, device=cuda), KN, beta=0.0)
    assert (dW == 0).all()
    with pytest.raises(q.QlmbError):               # K not a multiple of the scale group
        linear.linear_fwd(torch.zeros(4, 96, device=cuda), Q.d, Q.s, KN, 128)
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("M,K,N", [(300, 384, 640), (129, 640, 1152), (1000, 1408, 896), (70, 128, 384)])
def test_linear_widths_that_end_inside_a_column_tile(cuda, M, K, N):
    """Odd multiples of 128 on the output side: the last 256-column tile is half full."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    for lay in (KN, NK):
        Q, W = quantise(cuda, K, N, 31) if lay == KN else quantise(cuda, N, K, 31)
        Wm = W if lay == KN else W.T
        for dt in (torch.float32, torch.bfloat16):
            X, dY = torch.randn(M, K, device=cuda).to(dt), torch.randn(M, N, device=cuda).to(dt)
            Y, dX = linear.linear_fwd(X, Q.d, Q.s, lay, N), linear.linear_dgrad(dY, Q.d, Q.s, lay, K)
            assert Y.shape == (M, N) and rel(Y, X.float() @ Wm) < 8e-3, (lay, dt)
            assert dX.shape == (M, K) and rel(dX, dY.float() @ Wm.T) < 8e-3, (lay, dt)


@pytest.mark.parametrize("M", [1023, 1025, 2047, 4161, 8191])
def test_linear_wgrad_of_ragged_row_slices(cuda, M):
    """Rows that do not divide into the slices: the last slice ends early, or lies past the rows altogether."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    for K, N in ((256, 256), (384, 640)):
        X = torch.randn(M, K, device=cuda).bfloat16(); dY = torch.randn(M, N, device=cuda).bfloat16()
        for lay in (KN, NK):
            ref = X.float().T @ dY.float() if lay == KN else dY.float().T @ X.float()
            dW = torch.zeros(K * N, device=cuda)
            for beta in (0.0, 1.0):
                linear.linear_wgrad(dW, dY, X, lay, beta=beta)
                assert rel(dW.view(ref.shape), ref * (1.0 + beta)) < 1e-4, (K, N, lay, beta)


def test_linear_wgrad_of_slices_under_capture_and_on_two_streams(cuda):
    """The slices' partial sums are each call's own: the first sliced call of its size may be a captured one, a replay
    is not disturbed by larger calls since, and two streams may run such calls at once."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN
    K = N = 256

    def operands(M, seed):
        g = torch.Generator(device=cuda); g.manual_seed(seed)
        return tuple(torch.randn(M, n, device=cuda, generator=g).bfloat16() for n in (N, K)) + (torch.zeros(K * N, device=cuda),)
    linear.linear_wgrad(torch.zeros(K * N, device=cuda), *operands(100, 0)[:2], KN, beta=0.0)
    dy, x, dw = operands(5003, 1)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        linear.linear_wgrad(dw, dy, x, KN, beta=0.0)
    big = operands(40001, 2)
    linear.linear_wgrad(big[2], big[0], big[1], KN, beta=0.0)
    for _ in range(3):
        dw.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert rel(dw.view(K, N), x.float().T @ dy.float()) < 1e-4
    eager = torch.empty_like(dw)
    linear.linear_wgrad(eager, dy, x, KN, beta=0.0)
    assert torch.equal(eager, dw)
    streams, sets = [torch.cuda.Stream() for _ in range(2)], [operands(9001, 3), operands(9001, 4)]
    want = []
    for a in sets:
        linear.linear_wgrad(a[2], a[0], a[1], KN, beta=0.0)
        want.append(a[2].clone())
    outs = [[torch.empty_like(dw) for _ in range(50)] for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(50):
        for s, a, o in zip(streams, sets, outs):
            with torch.cuda.stream(s):
                linear.linear_wgrad(o[i], a[0], a[1], KN, beta=0.0)
    torch.cuda.synchronize()
    assert all(torch.equal(t, w) for o, w in zip(outs, want) for t in o)


@pytest.mark.parametrize("B", [1, 8, 64])
def test_gemv_decode(cuda, oracle, B):
    """Decode path (M = live slots <= 64).  fp32 activations: fp32 accumulation of exact dequantised weights (the
    digits are multiplied as 136 + d and the constant is taken out of the finished sums, which costs about five of
    the 24 mantissa bits), so the result agrees with the fp32 reference to round-off (3e-5).  bf16 activations with
    more than four slots run on warp-level MMAs with bf16(x * scale) operands: 8e-3."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    for K, N in ((768, 1536), (1536, 768), (768, 16384), (2048, 4096)):
        for lay in (KN, NK):
            Q, W = quantise(cuda, K, N, 5) if lay == KN else quantise(cuda, N, K, 5)
            Wm = W if lay == KN else W.T
            for dt in (torch.float32, torch.bfloat16):
                X = torch.randn(B, K, device=cuda).to(dt)
                Y = linear.gemv_decode(X, Q.d, Q.s, lay, N)
                ref = X.float() @ Wm
                assert rel(Y, ref) < (3e-5 if dt == torch.float32 else 8e-3), (K, N, lay, dt)
                assert torch.equal(Y, linear.gemv_decode(X, Q.d, Q.s, lay, N))      # deterministic
    # oracle on one case
    Q, W = quantise(cuda, 256, 384, 6)
    X = torch.randn(B, 256, device=cuda)
    Yo = oracle.linear_fwd(X.cpu().numpy(), Q.d.cpu().numpy(), Q.s.cpu().numpy(), 0, 384)
    assert rel(linear.gemv_decode(X, Q.d, Q.s, KN, 384), dev(Yo, cuda)) < 1e-5


@pytest.mark.parametrize("B", [1, 2, 3, 4, 5, 16, 17, 33])
def test_gemv_decode_edges(cuda, B):
    """K slices of unequal length, widths that end inside a column block, the smallest shape, and rows that start at an
    address no vector load can take."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN, NK
    for K, N in ((128, 128), (1664, 8320), (896, 2432), (640, 768)):
        for lay in (KN, NK):
            Q, W = quantise(cuda, K, N, 21) if lay == KN else quantise(cuda, N, K, 21)
            Wm = W if lay == KN else W.T
            for dt in (torch.float32, torch.bfloat16):
                X = torch.randn(B, K, device=cuda).to(dt)
                ref = X.float() @ Wm
                tol = 3e-5 if dt == torch.float32 else 8e-3
                assert rel(linear.gemv_decode(X, Q.d, Q.s, lay, N), ref) < tol, (K, N, lay, dt)
                if B <= 4:
                    odd = torch.empty(B * K + 1, device=cuda, dtype=dt)[1:].view(B, K).copy_(X)
                    assert rel(linear.gemv_decode(odd, Q.d, Q.s, lay, N), ref) < tol, (K, N, lay, dt)


@pytest.mark.parametrize("N", [768, 1024, 2304])
def test_gemv_decode_scales_at_any_group(cuda, N):
    """The scales of a matrix that follows another span may start at any float."""
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN
    K = 256
    Q, W = quantise(cuda, K, N, 5)
    for off in (1, 2, 3):
        s = torch.empty(Q.s.numel() + off, device=cuda)[off:].copy_(Q.s)
        for B in (5, 17, 40):
            X = torch.randn(B, K, device=cuda).bfloat16()
            assert torch.equal(linear.gemv_decode(X, Q.d, s, KN, N), linear.gemv_decode(X, Q.d, Q.s, KN, N)), (off, B)


def test_gemv_rejects_more_than_64_slots(cuda):
    import cudalm_c_b200 as q
    from cudalm_c_b200 import linear
    from cudalm_c_b200._lib import KN
    Q, W = quantise(cuda, 128, 128, 9)
    with pytest.raises(q.QlmbError):
        linear.gemv_decode(torch.zeros(65, 128, device=cuda), Q.d, Q.s, KN, 128)


@pytest.mark.parametrize("B", [1, 3, 8, 64])
def test_gemv_decode_res_norm_equals_the_separate_kernels(cuda, B):
    """wo + residual + norm of a decode step in one launch pair (dec_step, cudalm.cu:7188-7190): F is the same bf16
    values as the GEMV followed by the bf16 add; Fn agrees with the separate norm kernel to one bf16 rounding."""
    from cudalm_c_b200 import block, linear
    from cudalm_c_b200._lib import KN, check, lib, ptr, stream_ptr
    for K, N in ((768, 768), (1536, 2048)):
        Q, W = quantise(cuda, K, N, 12)
        X = torch.randn(B, K, device=cuda).to(torch.bfloat16)
        res = torch.randn(B, N, device=cuda).to(torch.bfloat16)
        gamma = 1.0 + 0.1 * torch.randn(N, device=cuda)
        F = torch.empty(B, N, dtype=torch.bfloat16, device=cuda); Fn = torch.empty_like(F)
        check(lib().qlmb_gemv_decode_res_norm(ptr(F), ptr(Fn), ptr(X), ptr(Q.d), ptr(Q.s), ptr(res), ptr(gamma), B, K, N,
                                              stream_ptr()))
        # the separate kernels of the same family (the plain qlmb_gemv_decode sums in another order for few rows)
        Y = torch.empty(B, N, dtype=torch.bfloat16, device=cuda)
        check(lib().qlmb_gemv_decode_stack(ptr(Y), ptr(X), ptr(Q.d), ptr(Q.s), 1, B, K, N, 1, stream_ptr()))
        Y += res
        assert torch.equal(F, Y)
        Yn, _ = block.rmsnorm_fwd(Y, gamma)
        assert rel(Fn, Yn) < 8e-3
        assert (Fn.float() - Yn.float()).abs().max() <= 2.0 ** -7 * Yn.float().abs().max()
        assert rel(F, X.float() @ W + res.float()) < 8e-3


@pytest.mark.parametrize("B", [1, 8, 64])
def test_gemv_decode_norm_stack(cuda, B):
    """The norm in front of the q, k, v projections applied while the rows are staged (e_rmsf + three g_ab,
    cudalm.cu:7176-7180): the same numbers as the norm kernel followed by the stacked GEMV, up to one bf16 rounding
    of a normalised input where the two row sums differ in their last bit."""
    from cudalm_c_b200 import block
    from cudalm_c_b200._lib import check, lib, ptr, stream_ptr
    K = N = 768
    Q, W = quantise(cuda, 3 * K, N, 14)                       # three [K, N] matrices one after the other
    X = torch.randn(B, K, device=cuda).to(torch.bfloat16)
    gamma = 1.0 + 0.1 * torch.randn(K, device=cuda)
    Y = torch.empty(3 * B, N, dtype=torch.bfloat16, device=cuda); Y2 = torch.empty_like(Y)
    check(lib().qlmb_gemv_decode_norm_stack(ptr(Y), ptr(X), ptr(gamma), ptr(Q.d), ptr(Q.s), 3, B, K, N, 1, stream_ptr()))
    Xn, _ = block.rmsnorm_fwd(X, gamma)
    check(lib().qlmb_gemv_decode_stack(ptr(Y2), ptr(Xn), ptr(Q.d), ptr(Q.s), 3, B, K, N, 1, stream_ptr()))
    assert rel(Y, Y2) < 2e-3
    assert (Y == Y2).float().mean() > 0.99
    ref = torch.cat([Xn.float() @ W[m * K:(m + 1) * K] for m in range(3)])
    assert rel(Y, ref) < 8e-3


@pytest.mark.parametrize("B", [1, 5, 64])
def test_dec_qkv_equals_the_separate_kernels(cuda, B):
    """Norm, q / k / v projections, rotation and cache append of a decode step in one launch pair (dec_step,
    cudalm.cu:7176-7183) against the chain of separate kernels: same rows, same cache contents, nothing else touched."""
    from cudalm_c_b200 import block
    from cudalm_c_b200._lib import check, lib, ptr, stream_ptr
    D, hd, Tm = 768, 64, 96
    H = D // hd
    Q, W = quantise(cuda, 3 * D, D, 21)
    X = torch.randn(B, D, device=cuda).to(torch.bfloat16)
    gamma = 1.0 + 0.1 * torch.randn(D, device=cuda)
    cosb, sinb = block.rope_tables(Tm, hd, device=cuda)
    pos = torch.randint(0, Tm, (B,), device=cuda, dtype=torch.int32)
    Kc = torch.full((B, Tm, D), 7.0, dtype=torch.bfloat16, device=cuda); Vc = Kc.clone()
    Y = torch.empty(3 * B, D, dtype=torch.bfloat16, device=cuda)
    check(lib().qlmb_dec_qkv(ptr(Y), ptr(Kc), ptr(Vc), ptr(X), ptr(gamma), ptr(Q.d), ptr(Q.s), ptr(cosb), ptr(sinb), ptr(pos),
                             B, D, hd, Tm, stream_ptr()))
    Y2 = torch.empty_like(Y)
    check(lib().qlmb_gemv_decode_norm_stack(ptr(Y2), ptr(X), ptr(gamma), ptr(Q.d), ptr(Q.s), 3, B, D, D, 1, stream_ptr()))
    pos2 = torch.cat([pos, pos])
    check(lib().qlmb_dec_rope(ptr(Y2), 1, ptr(cosb), ptr(sinb), ptr(pos2), 2 * B, H, hd, Tm, stream_ptr()))
    Kc2 = torch.full((B, Tm, D), 7.0, dtype=torch.bfloat16, device=cuda); Vc2 = Kc2.clone()
    check(lib().qlmb_dec_kv(ptr(Kc2), ptr(Vc2), ptr(Y2[B:2 * B]), ptr(Y2[2 * B:]), ptr(pos), B, Tm, D, stream_ptr()))
    assert rel(Y, Y2) < 1e-3 and (Y == Y2).float().mean() > 0.999
    assert torch.equal(Kc[torch.arange(B), pos.long()], Y[B:2 * B]) and torch.equal(Vc[torch.arange(B), pos.long()], Y[2 * B:])
    assert rel(Kc, Kc2) < 1e-3 and rel(Vc, Vc2) < 1e-3
    assert int((Kc != 7.0).sum()) <= B * D and int((Vc != 7.0).sum()) <= B * D


@pytest.mark.parametrize("M,D,KD,T", [(1, 256, 256, 1), (255, 384, 128, 85), (257, 512, 256, 200), (2100, 768, 768, 700), (640, 640, 640, 64)])
def test_qkv_projections_against_float64(cuda, M, D, KD, T):
    """The three projections with their rotation and both gradients, on one and on several row tiles, with widths that end inside
    a column tile and the fallback of a width of 128.  Bar: bf16 operands and results."""
    from cudalm_c_b200 import block, linear
    N = (D, KD, KD)
    ws, deq = zip(*[(lambda q, w: (q, w))(*quantise(cuda, D, n, 40 + i)) for i, n in enumerate(N)])
    ws = [(q.d, q.s) for q in ws]
    g = torch.Generator(device=cuda); g.manual_seed(7)
    rnd = lambda c: torch.randn(M, c, device=cuda, generator=g).to(torch.bfloat16)
    X, dq, dk, dv = rnd(D), rnd(D), rnd(KD), rnd(KD)
    cosb, sinb = block.rope_tables(T, 64, device=cuda)
    Y = linear.qkv_fwd(X, ws, KD, cosb, sinb, T)
    pos = torch.arange(M, device=cuda) % T
    c, s = cosb.double()[pos][:, None], sinb.double()[pos][:, None]
    for i in range(3):
        ref = X.double() @ deq[i].double()
        if i < 2:
            h = ref.view(M, N[i] // 64, 64)
            a, b = h[..., :32], h[..., 32:]
            ref = torch.cat([a * c - b * s, b * c + a * s], -1).reshape(M, N[i])
        assert float((Y[i].double() - ref).norm() / ref.norm()) < 1e-2
    for beta in (0.0, 1.0):
        dW = [torch.ones(D * n, device=cuda) for n in N]
        dX = linear.qkv_bwd(dW, dq, dk, dv, X, ws, cosb, sinb, T, beta=beta)
        ref = sum(d.double() @ w.double().T for d, w in zip((dq, dk, dv), deq))
        assert float((dX.double() - ref).norm() / ref.norm()) < 1e-2
        for w, d in zip(dW, (dq, dk, dv)):
            ref = X.double().T @ d.double()
            # bf16 products are exact in fp32: the sums' roundings alone
            assert float((w.view(D, -1).double() - beta - ref).norm() / ref.norm()) < 1e-5


@pytest.mark.parametrize("B,T,H,KV,win", [(2, 130, 4, 2, 0), (1, 64, 2, 2, 30), (1, 1, 2, 2, 0)])
def test_attention_gradients_rotated_back_on_the_way_out(cuda, B, T, H, KV, win):
    """Against the separate rotation, which rounds to bf16 once more."""
    from cudalm_c_b200 import attn, block
    g = torch.Generator(device=cuda); g.manual_seed(8)
    rnd = lambda c: torch.randn(B * T, c * 64, device=cuda, generator=g).to(torch.bfloat16)
    Q, K, V, dA = rnd(H), rnd(KV), rnd(KV), rnd(H)
    rot = block.rope_tables(T, 64, device=cuda)
    O, lse = attn.attn_fwd(Q, K, V, B, T, H, KV, win)
    dQ, dK, dV, _ = attn.attn_bwd(Q, K, V, O, dA, lse, B, T, H, KV, win)
    rQ, rK, rV, _ = attn.attn_bwd(Q, K, V, O, dA, lse, B, T, H, KV, win, rope=rot)
    assert torch.equal(dV, rV)
    for d, r, n in ((dQ, rQ, H), (dK, rK, KV)):
        block.rope(d, *rot, n, 64, T, back=True)
        assert float((d.float() - r.float()).norm()) <= 2 ** -7 * float(d.float().norm()) + 1e-6


@pytest.mark.parametrize("M,D", [(4608, 768), (1024, 1792), (1024, 2432)])
def test_joint_weight_gradients_under_capture_and_on_two_streams(cuda, M, D):
    """q, k and v's gradients in slices, where one matrix alone has scratch of its own (4608 rows: four slices that do not divide
    them) or none (1792 columns: no slices; 2432: one by one, two slices of the three are more than the scratch pool keeps): replays
    are not disturbed by larger calls since, two streams may run such calls at once."""
    from cudalm_c_b200 import block, linear
    cosb, sinb = block.rope_tables(64, 64, device=cuda)
    ws = [(lambda q: (q.d, q.s))(quantise(cuda, D, D, 60 + i)[0]) for i in range(3)]

    def call(m, seed):
        g = torch.Generator(device=cuda); g.manual_seed(seed)
        x, dq, dk, dv = (torch.randn(m, D, device=cuda, generator=g).bfloat16() for _ in range(4))
        return lambda dw: linear.qkv_bwd(dw, dq, dk, dv, x, ws, cosb, sinb, 64, beta=0.0)
    new = lambda: [torch.full((D * D,), -1.0, device=cuda) for _ in range(3)]
    one, two, dw = call(M, 1), call(M, 2), new()
    want = []
    for f in (one, two):
        want.append(new())
        f(want[-1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        one(dw)
    call(8 * 2048, 3)(new())                              # (rows that divide evenly: the largest shared piece of the shape)
    for _ in range(3):
        for t in dw:
            t.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(dw, want[0]))
    streams, outs = [torch.cuda.Stream() for _ in range(2)], [[new() for _ in range(20)] for _ in range(2)]
    torch.cuda.synchronize()
    for i in range(20):
        for s, f, o in zip(streams, (one, two), outs):
            with torch.cuda.stream(s):
                f(o[i])
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for o, w in zip(outs, want) for t in o for a, b in zip(t, w))
