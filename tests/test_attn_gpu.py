"""Flash attention (tcgen05, head dimension 64) through the C ABI against the reference's CPU
attention (cpu_kern.h:166-312, compiled from the reference's sources) on the same bf16-rounded inputs.
Bar: 1e-2 relative on outputs and gradients (P and dS are rounded to bf16 for the tensor core),
1e-3 absolute on the log-sum-exp."""
import numpy as np
import pytest
import torch

from oracle import loader

pytestmark = pytest.mark.gpu

SHAPES = [  # B, T, H, KV, win
    (2, 256, 4, 4, 0),
    (1, 200, 2, 1, 0),        # ragged sequence length, grouped-query heads
    (2, 384, 2, 2, 100),      # windowed
    (1, 1024, 2, 2, 0),
]


def rel(a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    return max(np.linalg.norm(a - b) / np.linalg.norm(b), np.abs(a - b).max() / np.abs(b).max())


def torch_attention(Q, K, V, B, T, H, KV, win, dA=None):
    """Plain fp64 attention with autograd: the stand-in when the compiled reference is not on the box."""
    Q, K, V = [torch.from_numpy(x).double().requires_grad_(True) for x in (Q, K, V)]
    q = Q.view(B, T, H, 64).transpose(1, 2)
    k = K.view(B, T, KV, 64).transpose(1, 2).repeat_interleave(H // KV, 1)
    v = V.view(B, T, KV, 64).transpose(1, 2).repeat_interleave(H // KV, 1)
    s = q @ k.transpose(-1, -2) / 8.0
    i = torch.arange(T)[:, None]; j = torch.arange(T)[None, :]
    mask = (j <= i) & ((j > i - win) if win > 0 else torch.ones_like(j <= i))
    s = s.masked_fill(~mask, float("-inf"))
    lse = torch.logsumexp(s, -1)
    O = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B * T, H * 64)
    if dA is None:
        return O.detach().numpy(), lse.detach().numpy()
    O.backward(torch.from_numpy(dA).double())
    return O.detach().numpy(), lse.detach().numpy(), Q.grad.numpy(), K.grad.numpy(), V.grad.numpy()


def inputs(B, T, H, KV, seed, cuda):
    g = torch.Generator(device="cpu"); g.manual_seed(seed)
    mk = lambda c: torch.randn(B * T, c * 64, generator=g).to(torch.bfloat16)
    Q, K, V = mk(H), mk(KV), mk(KV)
    return [x.to(cuda) for x in (Q, K, V)], [x.float().numpy() for x in (Q, K, V)]


@pytest.mark.parametrize("B,T,H,KV,win", SHAPES)
def test_attn_forward(cuda, B, T, H, KV, win):
    import cudalm_c_b200 as q
    from cudalm_c_b200 import attn
    ref = loader.reference()
    (Qd, Kd, Vd), (Qh, Kh, Vh) = inputs(B, T, H, KV, 3, cuda)
    O, lse = attn.attn_fwd(Qd, Kd, Vd, B, T, H, KV, win)
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    if ref is not None:
        Or, lr = ref.attn_fwd(Qh, Kh, Vh, B, T, H, KV, 64, win)
    else:
        Or, lr = torch_attention(Qh, Kh, Vh, B, T, H, KV, win)
    assert rel(O.float().cpu().numpy(), Or) < 1e-2
    assert np.abs(lse.cpu().numpy() - lr).max() < 1e-3


@pytest.mark.parametrize("B,T,H,KV,win", SHAPES)
def test_attn_backward(cuda, B, T, H, KV, win):
    import cudalm_c_b200 as q
    from cudalm_c_b200 import attn
    ref = loader.reference()
    (Qd, Kd, Vd), (Qh, Kh, Vh) = inputs(B, T, H, KV, 5, cuda)
    g = torch.Generator(device="cpu"); g.manual_seed(9)
    dA = torch.randn(B * T, H * 64, generator=g).to(torch.bfloat16)
    dAh = dA.float().numpy()
    if ref is not None:
        Or, lr = ref.attn_fwd(Qh, Kh, Vh, B, T, H, KV, 64, win)
        Ob = torch.from_numpy(Or).to(torch.bfloat16)
        dQr, dKr, dVr, drr = ref.attn_bwd(Qh, Kh, Vh, Ob.float().numpy(), dAh, lr, B, T, H, KV, 64, win)
    else:
        Or, lr, dQr, dKr, dVr = torch_attention(Qh, Kh, Vh, B, T, H, KV, win, dAh)
        Ob = torch.from_numpy(Or).to(torch.bfloat16)
        drr = None
    dQ, dK, dV, drow = attn.attn_bwd(Qd, Kd, Vd, Ob.to(cuda), dA.to(cuda), torch.from_numpy(lr.astype(np.float32)).to(cuda),
                                     B, T, H, KV, win)
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    if drr is not None:
        assert np.abs(drow.cpu().numpy() - drr).max() < 1e-3 * max(1.0, np.abs(drr).max())
    assert rel(dV.float().cpu().numpy(), dVr) < 1e-2
    assert rel(dK.float().cpu().numpy(), dKr) < 1e-2
    assert rel(dQ.float().cpu().numpy(), dQr) < 1e-2


@pytest.mark.parametrize("T", [1, 31, 33, 64, 65, 127, 129, 257])
@pytest.mark.parametrize("win", [0, 1, 64, 129])
def test_attn_edges(cuda, T, win):
    """Sequence lengths around the tiles of 32, 64 and 128 rows, windows that end inside them, and scores that grow along the
    keys, so that most steps of a row bring a new maximum and O is rescaled.  The bar is that of the tests above: P and dS are
    bf16 (2^-9 each), O and the gradients are rounded once more, D is made of the rounded O."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import attn
    B, H, KV = 2, 2, 1
    _, (Qh, Kh, Vh) = inputs(B, T, H, KV, 11, cuda)
    Kh = Kh * np.tile(1.0 + 2.0 * np.arange(T) / T, B)[:, None].astype(np.float32)
    Kh = torch.from_numpy(Kh).to(torch.bfloat16).float().numpy()
    g = torch.Generator(device="cpu"); g.manual_seed(13)
    dA = torch.randn(B * T, H * 64, generator=g).to(torch.bfloat16)
    Or, lr, dQr, dKr, dVr = torch_attention(Qh, Kh, Vh, B, T, H, KV, win, dA.float().numpy())
    Qd, Kd, Vd = [torch.from_numpy(x).to(torch.bfloat16).to(cuda) for x in (Qh, Kh, Vh)]
    O, lse = attn.attn_fwd(Qd, Kd, Vd, B, T, H, KV, win)
    dQ, dK, dV, _ = attn.attn_bwd(Qd, Kd, Vd, O, dA.to(cuda), lse, B, T, H, KV, win)
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    norm = lambda a, b: float(np.linalg.norm(a.float().cpu().numpy().astype(np.float64) - b) / max(np.linalg.norm(b), 1e-3))
    assert norm(O, Or) < 1e-2 and np.abs(lse.cpu().numpy() - lr).max() < 1e-3
    assert norm(dV, dVr) < 1e-2
    if T > 1 and win != 1:
        assert norm(dQ, dQr) < 1e-2 and norm(dK, dKr) < 1e-2
    else:
        # one visible key: dS is zero in exact arithmetic, what is left is the rounding of O inside D, at most 2^-8 of the sum of
        # its terms' absolute values, times a component of K (or of Q, from each of the key's heads) and 1/8
        f = lambda t: t.double().cpu().abs().view(B * T, -1, 64)
        d = 2 ** -8 * (f(dA) * f(O)).sum(-1)
        assert bool((f(dQ).amax(-1) <= d * f(Kd).max() / 8).all()) and bool((f(dK).amax(-1) <= d.sum(-1, keepdim=True) * f(Qd).max() / 8).all())


@pytest.mark.parametrize("B,T,H,KV,win", [(1, 300, 4, 1, 0), (2, 129, 8, 1, 50), (1, 64, 8, 2, 0), (75, 100, 8, 4, 0), (1, 200, 6, 2, 0)])
def test_attn_gradients_of_grouped_heads(cuda, B, T, H, KV, win):
    """Two, four and eight query heads on a key/value head, whose gradients a cluster adds, three heads and a grid that fills the
    device, which one CTA walks; with and without the rotation undone.  Bars as above."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import attn, block
    (Qd, Kd, Vd), (Qh, Kh, Vh) = inputs(B, T, H, KV, 21, cuda)
    g = torch.Generator(device="cpu"); g.manual_seed(23)
    dA = torch.randn(B * T, H * 64, generator=g).to(torch.bfloat16)
    Or, lr, dQr, dKr, dVr = torch_attention(Qh, Kh, Vh, B, T, H, KV, win, dA.float().numpy())
    O, lse = attn.attn_fwd(Qd, Kd, Vd, B, T, H, KV, win)
    dQ, dK, dV, drow = attn.attn_bwd(Qd, Kd, Vd, O, dA.to(cuda), lse, B, T, H, KV, win)
    again = attn.attn_bwd(Qd, Kd, Vd, O, dA.to(cuda), lse, B, T, H, KV, win)
    rot = block.rope_tables(T, 64, device=cuda)
    rQ, rK, rV, _ = attn.attn_bwd(Qd, Kd, Vd, O, dA.to(cuda), lse, B, T, H, KV, win, rope=rot)
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assert all(torch.equal(a, b) for a, b in zip((dQ, dK, dV, drow), again)) and torch.equal(rV, dV)
    norm = lambda a, b: float(np.linalg.norm(a.float().cpu().numpy().astype(np.float64) - b) / np.linalg.norm(b))
    assert norm(O, Or) < 1e-2 and norm(dQ, dQr) < 1e-2 and norm(dK, dKr) < 1e-2 and norm(dV, dVr) < 1e-2
    ref = (torch.from_numpy(Or).view(B, T, H, 64) * dA.double().view(B, T, H, 64)).sum(-1).permute(0, 2, 1).numpy()
    assert np.abs(drow.cpu().numpy() - ref).max() < 2 ** -7 * np.abs(ref).max()
    block.rope(dK, *rot, KV, 64, T, back=True)
    assert float((dK.float() - rK.float()).norm()) <= 2 ** -7 * float(rK.float().norm())


@pytest.mark.parametrize("B,T,H,KV,win,rope", [(2, 200, 4, 4, 0, False), (1, 130, 8, 2, 40, True), (3, 64, 2, 1, 0, True)])
@pytest.mark.parametrize("place", ["Q", "dA", "O"])
def test_dq_in_the_place_of_an_input(cuda, B, T, H, KV, win, rope, place):
    """dQ over Q, dA or O: the bits of separate buffers, with one CTA and with a cluster for dK and dV."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import attn, block
    from cudalm_c_b200._lib import ptr, stream_ptr
    g = torch.Generator(device=cuda); g.manual_seed(31)
    rnd = lambda c: torch.randn(B * T, c * 64, device=cuda, generator=g).to(torch.bfloat16)
    t = dict(Q=rnd(H), K=rnd(KV), V=rnd(KV), dA=rnd(H))
    t["O"], lse = attn.attn_fwd(t["Q"], t["K"], t["V"], B, T, H, KV, win)
    rot = block.rope_tables(T, 64, device=cuda) if rope else None
    want = attn.attn_bwd(t["Q"], t["K"], t["V"], t["O"], t["dA"], lse, B, T, H, KV, win, rope=rot)
    dK, dV, drow = torch.empty_like(t["K"]), torch.empty_like(t["V"]), torch.empty_like(want[3])
    args = [ptr(x) for x in (t[place], dK, dV, drow, t["Q"], t["K"], t["V"], t["O"], t["dA"], lse)]
    if rope:
        q.check(q.lib().qlmb_attn_bwd_rope(*args, ptr(rot[0]), ptr(rot[1]), B, T, H, KV, 64, win, stream_ptr()))
    else:
        q.check(q.lib().qlmb_attn_bwd(*args, B, T, H, KV, 64, win, stream_ptr()))
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assert all(torch.equal(a, b) for a, b in zip((t[place], dK, dV, drow), want))
