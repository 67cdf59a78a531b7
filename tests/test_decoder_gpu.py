"""The decoder (Dec / dec_prefill / dec_step, cudalm.cu:7020-7212) checked the way the reference's own
`decheck` does (cudalm.cu:7233-7285): logits of the cached one-token steps against the full forward over the
same tokens (teacher forcing), two slots with different prefixes; bar as there: worst |dlogit| < 5e-2 and
the same arg-max at every position."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_decoder_matches_full_forward(cuda):
    import cudalm_c_b200 as q
    from cudalm_c_b200 import block, model
    cfg = model.Config(L=2, D=128, H=2, KV=2, hd=64, E=4, K=2, F=128, V=256, T=128, B=2)
    m = model.QlmModel(cfg, cuda, seed=5)
    g = torch.Generator(device="cpu"); g.manual_seed(1)
    B, n, k = 2, 40, 8
    ids = torch.randint(0, cfg.V, (B, n + k), generator=g, dtype=torch.int32).to(cuda)
    # reference: the full forward over prompt + continuation
    full = model.Decoder(m, B, 64)
    moes = [full._moe(l, B * (n + k)) for l in range(cfg.L)]
    fn = m.forward(ids.reshape(-1).contiguous(), B=B, T=n + k, moes=moes)
    emb_bf, _ = block.cast_bf16(m.emb)
    ref = block.gemm_nt(fn, emb_bf, torch.float32).view(B, n + k, cfg.V)
    dec = model.Decoder(m, B, 64)
    lg = dec.prefill(ids[:, :n].contiguous())
    worst, agree, tot = 0.0, 0, 0

    def cmp(got, want):
        nonlocal worst, agree, tot
        worst = max(worst, float((got - want).abs().max()))
        agree += int((got.argmax(-1) == want.argmax(-1)).sum()); tot += got.shape[0]

    cmp(lg, ref[:, n - 1])
    for j in range(k):
        dec.tok.copy_(ids[:, n + j])
        lg = dec.step(advance=False)
        dec.advance()
        cmp(lg, ref[:, n + j])
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assert int(dec.pos[0]) == n + k
    assert worst < 5e-2 and agree == tot, (worst, agree, tot)
    # greedy continuation runs without host input and picks the arg-max
    dec.step()
    assert torch.equal(dec.otok.long(), dec.logits.argmax(-1))


def test_slot_past_its_cache_is_reported_not_written(cuda):
    """Positions live on the device: a slot whose position equals the cache length must not touch the cache, the
    score buffer or the rotation tables.  The kernels skip it and leave error 201 in the device error word."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    cfg = model.Config(L=1, D=128, H=2, KV=2, hd=64, E=4, K=2, F=128, V=256, T=64, B=2)
    m = model.QlmModel(cfg, cuda, seed=6)
    dec = model.Decoder(m, 2, 32)
    g = torch.Generator(device="cpu"); g.manual_seed(2)
    ids = torch.randint(0, cfg.V, (2, 8), generator=g, dtype=torch.int32).to(cuda)
    dec.prefill(ids)
    dec.step()
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    K0, V0 = dec.K[0].clone(), dec.V[0].clone()
    dec.pos2.fill_(32)                                   # one past the last cache position
    dec.step(advance=False)
    torch.cuda.synchronize()
    assert q.lib().qlmb_check_device(None) == 4          # QLMB_E_DEVICE
    assert b"error code 201" in q.lib().qlmb_last_error()
    assert torch.equal(K0, dec.K[0]) and torch.equal(V0, dec.V[0])
    dec.pos2.fill_(9)
    dec.step()                                           # the context is intact: the next step runs
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    # the stand-alone rotation has the same guard: a position outside its tables leaves the row alone and is reported
    from cudalm_c_b200._lib import ptr, stream_ptr
    row = torch.randn(2, cfg.D, device=cuda).to(torch.bfloat16); keep = row.clone()
    pos = torch.tensor([3, 32], dtype=torch.int32, device=cuda)
    q.check(q.lib().qlmb_dec_rope(ptr(row), 1, ptr(dec.cosb), ptr(dec.sinb), ptr(pos), 2, cfg.H, cfg.hd, 32, stream_ptr()))
    torch.cuda.synchronize()
    assert q.lib().qlmb_check_device(None) == 4 and b"error code 201" in q.lib().qlmb_last_error()
    assert torch.equal(row[1], keep[1]) and not torch.equal(row[0], keep[0])


CHAIN = [(9, 256, 4, 2, 128), (17, 256, 2, 2, 256), (64, 768, 12, 2, 256), (12, 1152, 18, 2, 128)]      # B, D, KV, experts = choices, F


@pytest.mark.parametrize("B,D,KV,E,F", CHAIN)
def test_chain_matches_full_forward(cuda, B, D, KV, E, F):
    """Steps of more than eight slots (and of a width beyond the one-launch form) go through the chain of separate operators:
    the check above for them, slots at different positions.  Every token takes every expert, so that no near-tie of two
    router logits decides between experts."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import block, model
    cfg = model.Config(L=2, D=D, H=D // 64, KV=KV, hd=64, E=E, K=E, F=F, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=5)
    g = torch.Generator(device=cuda); g.manual_seed(B)
    n, k = 21, 3
    ids = torch.randint(0, cfg.V, (B, n + k), generator=g, dtype=torch.int32, device=cuda)
    dec = model.Decoder(m, B, 48)
    assert dec._step_plan() is None
    fn = m.forward(ids.reshape(-1).contiguous(), B=B, T=n + k, moes=[dec._moe(l, B * (n + k)) for l in range(cfg.L)])
    ref = block.gemm_nt(fn, block.cast_bf16(m.emb)[0], torch.float32).view(B, n + k, cfg.V)
    back = torch.arange(B, device=cuda, dtype=torch.int32) % 5             # slot b has n - back[b] tokens cached
    dec.prefill(ids[:, :n].contiguous())
    dec.pos2.sub_(back.repeat(2))
    rows = torch.arange(B, device=cuda)
    for j in range(k):
        at = (dec.pos + 0).long()
        dec.tok.copy_(ids[rows, at])
        lg = dec.step(advance=False)
        dec.advance()
        want = ref[rows, at]
        assert float((lg - want).abs().max()) < 5e-2
        assert float((lg.argmax(-1) == want.argmax(-1)).float().mean()) > 0.98
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("B,D,KV,E,F", CHAIN)
def test_chain_skips_a_slot_past_its_cache(cuda, B, D, KV, E, F):
    """One slot's position outside the cache: reported, its cache rows untouched, the other slots' logits the same bits."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    cfg = model.Config(L=2, D=D, H=D // 64, KV=KV, hd=64, E=E, K=E, F=F, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=6)
    dec = model.Decoder(m, B, 32)
    g = torch.Generator(device=cuda); g.manual_seed(B)
    dec.prefill(torch.randint(0, cfg.V, (B, 11), generator=g, dtype=torch.int32, device=cuda))
    good = dec.step(advance=False).clone()
    q.check(q.lib().qlmb_check_device(None))
    others = torch.arange(B, device=cuda) != 3
    for bad in (32, -1, 2 ** 30):
        dec.pos2[3] = bad; dec.pos2[B + 3] = bad
        keep = [t[3].clone() for t in dec.K + dec.V]
        got = dec.step(advance=False)
        torch.cuda.synchronize()
        assert q.lib().qlmb_check_device(None) == 4 and b"error code 201" in q.lib().qlmb_last_error()
        assert all(torch.equal(t[3], u) for t, u in zip(dec.K + dec.V, keep))
        assert torch.equal(got[others], good[others])
    dec.pos2[3] = 11; dec.pos2[B + 3] = 11
    assert torch.equal(dec.step(advance=False), good)
    q.check(q.lib().qlmb_check_device(None))


def test_sampler_topk_topp_temperature(cuda):
    """k_dec_sample (cudalm.cu:7048-7108) against a float64 restatement of its algorithm: arg-max and
    log-probability, the top-k / top-p cut, and the pick that the (seed, step) hash selects from the tempered
    distribution.  The device adds float32 exponentials, so the pick is accepted when the hashed number falls
    within 1e-4 of the pick's interval of the cumulative distribution."""
    import numpy as np
    import cudalm_c_b200 as q
    from cudalm_c_b200._lib import check, lib, ptr, stream_ptr
    rng = np.random.default_rng(0)
    V, B = 16384, 12
    lg = (rng.standard_normal((B, V)) * 2.5).astype(np.float32)
    lg[3, 100] = lg[3].max() + 3.0                               # a dominant token
    dt = np.dtype(dict(names=["temp", "top_p", "top_k", "seed", "step"], formats=["<f4", "<f4", "<i4", "<u8", "<i4"],
                       offsets=[0, 4, 8, 16, 24], itemsize=32))
    prm = np.zeros(B, dt)
    cases = [(0.0, 1.0, 0), (1.0, 1.0, 1), (1.0, 1.0, 0), (0.7, 0.9, 40), (1.3, 0.5, 0), (0.5, 1.0, 5),
             (1.0, 0.95, 200), (2.0, 0.99, 0), (0.9, 0.8, 3), (1.0, 0.3, 0), (0.8, 1.0, 1000), (1.5, 0.7, 64)]
    for b, (temp, top_p, top_k) in enumerate(cases):
        prm[b] = (temp, top_p, top_k, 1234 + 77 * b, 5 + b)
    d_lg = torch.from_numpy(lg).to(cuda)
    d_prm = torch.from_numpy(prm.view(np.uint8).reshape(B, 32).copy()).to(cuda)
    out = torch.zeros(B, dtype=torch.int32, device=cuda); lp = torch.zeros(B, device=cuda)
    check(lib().qlmb_dec_sample(ptr(out), ptr(lp), ptr(d_lg), ptr(d_prm), B, V, stream_ptr()))
    torch.cuda.synchronize()
    out, lp = out.cpu().numpy(), lp.cpu().numpy()
    M64 = (1 << 64) - 1
    for b, (temp, top_p, top_k) in enumerate(cases):
        l = lg[b].astype(np.float64)
        ls = l.max() + np.log(np.exp(l - l.max()).sum())
        assert abs(lp[b] - (l[out[b]] - ls)) < 1e-3
        if temp <= 0 or top_k == 1:
            assert out[b] == int(np.argmax(l))
            continue
        th = l.max() - 30.0
        while (lg[b] >= np.float32(th)).sum() > 2048:
            th = 0.5 * (th + l.max())
        idx = np.nonzero(lg[b] >= np.float32(th))[0]
        order = idx[np.lexsort((idx, -l[idx]))]                   # value descending, index ascending
        sv = l[order]
        k = min(top_k, len(order)) if top_k > 0 else len(order)
        e = np.exp(sv[:k] - sv[0])
        if top_p < 1.0:
            c = np.cumsum(e / e.sum())
            hit = np.nonzero(c >= top_p - 1e-6)[0]
            k_lo = int(np.nonzero(c >= top_p + 1e-6)[0][0]) + 1 if (c >= top_p + 1e-6).any() else k
            k = int(hit[0]) + 1 if len(hit) else k
        else:
            k_lo = k
        h = ((1234 + 77 * b) * 0x9E3779B97F4A7C15 + (5 + b + 1) * 0xD1B54A32D192ED03) & M64
        h ^= h >> 30; h = (h * 0xBF58476D1CE4E5B9) & M64; h ^= h >> 27; h = (h * 0x94D049BB133111EB) & M64; h ^= h >> 31
        u01 = (h >> 40) / 16777216.0
        ok = False
        for kk in {k, k_lo}:                                      # a cumulative sum within rounding of top_p may cut one later
            w = np.exp((sv[:kk] - sv[0]) / temp)
            cum = np.cumsum(w) / w.sum()
            pos = np.nonzero(order[:kk] == out[b])[0]
            if len(pos):
                i = int(pos[0])
                lo = cum[i - 1] if i else 0.0
                ok |= lo - 1e-4 <= u01 <= cum[i] + 1e-4
        assert ok, (b, cases[b], int(out[b]))
    q.check(q.lib().qlmb_check_device(None))


def test_one_launch_step_skips_a_slot_past_its_cache(cuda):
    """The same for up to eight slots, which take one launch."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    cfg = model.Config(L=2, D=256, H=4, KV=4, hd=64, E=8, K=2, F=256, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=6)
    dec = model.Decoder(m, 5, 32)
    g = torch.Generator(device=cuda); g.manual_seed(1)
    dec.prefill(torch.randint(0, cfg.V, (5, 11), generator=g, dtype=torch.int32, device=cuda))
    assert dec._step_plan() is not None
    good = dec.step(advance=False).clone()
    for bad in (32, -1, 2 ** 30):
        dec.pos2[3] = bad; dec.pos2[8] = bad
        keep = [t[3].clone() for t in dec.K + dec.V]
        got = dec.step(advance=False)
        torch.cuda.synchronize()
        assert q.lib().qlmb_check_device(None) == 4 and b"error code 201" in q.lib().qlmb_last_error()
        assert all(torch.equal(t[3], u) for t, u in zip(dec.K + dec.V, keep))
        assert torch.equal(got[[0, 1, 2, 4]], good[[0, 1, 2, 4]])
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("win", [0, 100])
def test_decode_attention_with_values_at_any_pair(cuda, win):
    """A value cache that starts at a 4-byte address: the same bits as one that starts at 16."""
    import cudalm_c_b200 as q
    from cudalm_c_b200._lib import ptr, stream_ptr
    B, Tm, H, KV = 6, 300, 8, 4
    Q = torch.randn(B, H * 64, device=cuda).bfloat16()
    K, V = (torch.randn(B, Tm, KV * 64, device=cuda).bfloat16() for _ in range(2))
    pos = torch.tensor([0, 1, 63, 64, 200, 299], dtype=torch.int32, device=cuda)
    outs = []
    for off in (0, 2, 4, 6):
        v = torch.empty(V.numel() + off, dtype=V.dtype, device=cuda)[off:].view_as(V).copy_(V)
        O = torch.empty_like(Q)
        q.check(q.lib().qlmb_dec_attn(ptr(O), ptr(Q), ptr(K), ptr(v), ptr(pos), win, B, Tm, H, KV, 64, stream_ptr()))
        outs.append(O)
    assert all(torch.equal(o, outs[0]) for o in outs)
    for b in range(B):
        t = int(pos[b]); lo = max(0, t - win + 1) if win else 0
        k, v = (c[b, lo:t + 1].float().view(-1, KV, 64).repeat_interleave(H // KV, 1) for c in (K, V))
        p = torch.softmax(torch.einsum("hd,shd->hs", Q[b].float().view(H, 64), k) / 8.0, 1)
        ref = torch.einsum("hs,shd->hd", p, v).reshape(-1)
        assert float((outs[0][b].float() - ref).norm() / ref.norm()) < 1e-2


def test_step_after_tensors_were_replaced(cuda):
    """A caller's own token and position tensors, caches and gains in the place of the decoder's: the next step works on
    them, also one at an address that only the chain takes; a step captured before keeps its own."""
    from cudalm_c_b200 import model
    cfg = model.Config(L=2, D=256, H=4, KV=4, hd=64, E=8, K=2, F=256, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=3)

    def fresh():
        d = model.Decoder(m, 2, 64)
        g = torch.Generator(device=cuda); g.manual_seed(5)
        d.prefill(torch.randint(0, cfg.V, (2, 5), dtype=torch.int32, device=cuda, generator=g))
        return d
    tok = torch.tensor([17, 401], dtype=torch.int32, device=cuda)
    d = fresh()
    d.tok.copy_(tok)
    want = d.step(advance=False).clone()
    d = fresh()
    first = d.step(advance=False).clone()
    assert not torch.equal(first, want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        d.step(advance=False)
    captured = (d.tok, list(d.K), list(d.V))
    d.tok = tok.clone()                                                      # by value in the launch
    assert torch.equal(d.step(advance=False), want)
    d.K = [t.clone() for t in d.K]                                           # in the table
    for t in d.K:
        t[:, :5].neg_()
    other = d.step(advance=False).clone()
    assert not torch.equal(other, want)
    for t in d.K:
        t[:, :5].neg_()

    def values(off):
        return [torch.empty(t.numel() + off, dtype=t.dtype, device=cuda)[off:].view_as(t).copy_(t) for t in captured[2]]
    d.V = values(8)
    assert torch.equal(d.step(advance=False), want)
    d.V = values(2)                                                          # not on 16 bytes: the chain
    assert d._step_plan() is None
    got = d.step(advance=False)
    assert float((got - want).norm() / want.norm()) < 2e-2
    d.V = values(16)
    with torch.cuda.graph(torch.cuda.CUDAGraph()):                           # no address can be uploaded here: the chain
        assert d._step_plan() is None
        d.step(advance=False)
    assert torch.equal(d.step(advance=False), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(d.logits, first)


def test_one_launch_step_reports_a_misaligned_table(cuda):
    """A pointer of the device table that its loads cannot take: reported, nothing read through it, nothing written; the
    next step runs as usual."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    from cudalm_c_b200._lib import stream_ptr
    cfg = model.Config(L=2, D=256, H=4, KV=4, hd=64, E=8, K=2, F=256, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=3)
    d = model.Decoder(m, 2, 64)
    d.prefill(torch.randint(0, cfg.V, (2, 5), dtype=torch.int32, device=cuda))
    plan = d._step_plan()
    q.check(q.lib().qlmb_dec_step(plan, stream_ptr()))
    want = d.fn.clone()
    table, = d._tables.values()
    for l, word, off in ((0, 14, 4), (1, 4, 8), (1, 17, 2), (1, 22, 1), (0, 9, None)):
        keep = table[l, word].clone()
        table[l, word] = 0 if off is None else keep + off
        d.fn.fill_(7.0)
        q.check(q.lib().qlmb_dec_step(plan, stream_ptr()))
        assert q.lib().qlmb_check_device(None) != 0 and b"site 304, block %d, detail %d" % (l, word) in q.lib().qlmb_last_error()
        assert bool((d.fn == 7.0).all())
        table[l, word] = keep
        q.check(q.lib().qlmb_dec_step(plan, stream_ptr()))
        q.check(q.lib().qlmb_check_device(None))
        assert torch.equal(d.fn, want)


@pytest.mark.parametrize("B,D,KV,E,K,F,fill,Tm", [
    (1, 256, 4, 8, 2, 256, 1, 64),          # one key before the new one
    (1, 768, 12, 32, 2, 1536, 255, 640),    # the last key of a 256-key pass is the new one
    (2, 640, 2, 8, 1, 384, 256, 640),       # grouped heads, a column tile that is half empty, a second pass
    (3, 128, 2, 4, 4, 128, 40, 64),         # every expert, one row slice
    (8, 1024, 16, 32, 3, 640, 20, 32),      # 24 routed slots, experts with several slots, the widest model
    (3, 768, 12, 32, 2, 1536, 640, 1024),   # two rows a task, the last of them alone; buffers of keys used a second time
    (4, 768, 12, 32, 2, 512, 518, 1024),    # two rows a task; positions on both sides of 512
])
def test_one_launch_step_equals_the_chain(cuda, B, D, KV, E, K, F, fill, Tm):
    """qlmb_dec_step (up to eight slots) against the chain of separate operators: the same experts and the same cache rows
    up to a bf16 rounding, the final norm's output within the rounding noise of bf16 activations; bit-reproducible."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    from cudalm_c_b200._lib import stream_ptr
    cfg = model.Config(L=2, D=D, H=D // 64, KV=KV, hd=64, E=E, K=K, F=F, V=512, T=max(fill, 64), B=1)
    m = model.QlmModel(cfg, cuda, seed=3)
    d = model.Decoder(m, B, Tm)
    g = torch.Generator(device=cuda); g.manual_seed(B)
    d.prefill(torch.randint(0, cfg.V, (B, fill), generator=g, dtype=torch.int32, device=cuda))
    pos = torch.randint((fill + 1) // 2, fill + 1, (B,), generator=g, dtype=torch.int32, device=cuda)
    pos[0] = fill
    d.pos2.copy_(pos.repeat(2))
    plan = d._step_plan()
    assert plan is not None
    before = [t.clone() for t in d.K + d.V]
    want = d._layers_chain().float()
    experts = [mo.member("assign", (K, B), torch.int32).clone() for mo in d.moes]
    caches = [t.clone() for t in d.K + d.V]
    for t, b in zip(d.K + d.V, before):
        t.copy_(b)
    outs = []
    for _ in range(2):
        q.check(q.lib().qlmb_dec_step(plan, stream_ptr()))
        outs.append(d.fn.float().clone())
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assert torch.equal(*outs)
    # a near-tie of two router logits may fall the other way in one slot of a batch; every other slot is held to the bound:
    # some twenty bf16 roundings in two layers, each of at most 2^-9 and together 2^-9 sqrt(20 / 3) = 5e-3 by their root mean
    # square, times four for the largest of the slots
    same = torch.stack([(e == mo.member("assign", (K, B), torch.int32)).all(0) for e, mo in zip(experts, d.moes)]).all(0)
    assert int((~same).sum()) <= (B > 2)
    err = (outs[0] - want).norm(dim=1) / want.norm(dim=1)
    assert float(err[same].max()) < 2e-2, err.tolist()
    for t, c, b in zip(d.K + d.V, caches, before):
        assert float((t.float() - c.float()).abs().max()) < 2e-2
        assert ((t != b).flatten(2).any(-1).sum(1) <= 1).all()              # at most the slot's own row changed


@pytest.mark.parametrize("B,D,KV,E,K,F,fill,Tm", [
    (9, 768, 12, 32, 2, 1536, 255, 640),    # the smallest; an attention item per CTA
    (12, 1024, 16, 32, 2, 640, 20, 64),     # two items of a CTA, rows' owners among them; nearly all of the rows' room
    (16, 640, 10, 8, 2, 384, 600, 640),     # 32 routed slots, four of each expert, several passes of keys
    (32, 256, 2, 8, 1, 128, 40, 64),        # one choice a slot; grouped heads
    (17, 512, 8, 32, 2, 384, 90, 128),      # 34 routed slots: two of them in the second half of the list
    (32, 384, 6, 16, 2, 256, 30, 64),       # 64, most experts in both halves
    (21, 128, 2, 16, 3, 128, 300, 640),     # 63 of three choices, one row slice
])
def test_one_launch_step_of_more_slots_equals_the_chain(cuda, B, D, KV, E, K, F, fill, Tm):
    """The same above eight slots, where the attention's items outnumber the CTAs or share them with the rows' owners."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    from cudalm_c_b200._lib import stream_ptr
    cfg = model.Config(L=2, D=D, H=D // 64, KV=KV, hd=64, E=E, K=K, F=F, V=512, T=max(fill, 64), B=1)
    m = model.QlmModel(cfg, cuda, seed=3)
    d = model.Decoder(m, B, Tm)
    g = torch.Generator(device=cuda); g.manual_seed(B)
    d.prefill(torch.randint(0, cfg.V, (B, fill), generator=g, dtype=torch.int32, device=cuda))
    pos = torch.randint((fill + 1) // 2, fill + 1, (B,), generator=g, dtype=torch.int32, device=cuda)
    pos[0] = fill
    d.pos2.copy_(pos.repeat(2))
    plan = d._step_plan()
    assert plan is not None
    before = [t.clone() for t in d.K + d.V]
    want = d._layers_chain().float()
    chain = [(mo.member("assign", (K, B), torch.int32).clone(), mo.member("rt", (B, E), torch.float32).clone()) for mo in d.moes]
    caches = [t.clone() for t in d.K + d.V]
    for t, b in zip(d.K + d.V, before):
        t.copy_(b)
    outs = []
    for _ in range(3):
        q.check(q.lib().qlmb_dec_step(plan, stream_ptr()))
        outs.append(d.fn.float().clone())
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    # the bound of the test above, 2e-2 of the norm, for the slots with the same experts.  A slot may differ from the first
    # layer on where two of its logits are nearer than their noise: 5e-3 of a logit's root mean square each (the same
    # roundings), sqrt(2) for a difference, times four
    same = torch.ones(B, dtype=torch.bool, device=cuda)
    for (e, rt), mo in zip(chain, d.moes):
        now = (e == mo.member("assign", (K, B), torch.int32)).all(0)
        top = rt.sort(dim=1, descending=True).values[:, :K + 1]
        gap = (top[:, :-1] - top[:, 1:]).min(1).values / rt.pow(2).mean(1).sqrt()
        assert bool((now | ~same | (gap < 4 * 2 ** 0.5 * 5e-3)).all()), gap[~now].tolist()
        same &= now
    assert int(same.sum()) >= B // 2
    err = (outs[0] - want).norm(dim=1) / want.norm(dim=1)
    assert float(err[same].max()) < 2e-2, err.tolist()
    for i, (t, c, b) in enumerate(zip(d.K + d.V, caches, before)):
        keep = same if i % cfg.L else torch.ones_like(same)                     # the first layer's rows come before any router
        assert float((t.float() - c.float())[keep].abs().max()) < 2e-2
        assert ((t != b).flatten(2).any(-1).sum(1) <= 1).all()              # at most the slot's own row changed


def test_shapes_of_the_one_launch_step(cuda):
    """Above eight slots the form is left to shapes with few slots per expert, moderate experts and rows that shared memory holds."""
    import cudalm_c_b200 as q
    takes = [bool(q.lib().qlmb_dec_step_bytes(B, 64, D, D // 64, D // 64, F, E, K))
             for B, D, F, E, K in ((8, 1024, 8192, 8, 4), (9, 1024, 256, 8, 2), (12, 1024, 2048, 8, 2), (12, 1024, 2176, 8, 2), (13, 1024, 256, 32, 2),
                                   (16, 768, 256, 8, 2), (16, 768, 256, 7, 2), (25, 512, 256, 32, 2), (26, 512, 256, 32, 2), (32, 256, 256, 16, 2), (32, 256, 256, 15, 2),
                                   (22, 256, 256, 32, 3), (32, 256, 256, 8, 1), (33, 256, 256, 32, 1), (8, 256, 256, 8, 5))]
    assert takes == [True, True, True, False, False, True, False, True, False, True, False, False, True, False, False]


@pytest.mark.parametrize("L", [1, 2, 3, 4])
def test_one_launch_steps_in_a_row_and_a_workspace_of_several_shapes(cuda, L):
    """What the CTAs hand to one another lies in three slots used in turn across layers and launches, whatever the number of
    layers leaves them at, and a workspace may go to another shape and come back: the same bits at every launch."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import model
    from cudalm_c_b200._lib import ptr, stream_ptr
    cfg = model.Config(L=L, D=256, H=4, KV=2, hd=64, E=8, K=2, F=384, V=512, T=64, B=1)
    m = model.QlmModel(cfg, cuda, seed=3)
    g = torch.Generator(device=cuda); g.manual_seed(L)
    decs, want = [], []
    for B in (1, 3, 8):
        d = model.Decoder(m, B, 64)
        d.prefill(torch.randint(0, cfg.V, (B, 20), generator=g, dtype=torch.int32, device=cuda))
        q.check(q.lib().qlmb_dec_step(d._step_plan(), stream_ptr()))
        decs.append(d)
        want.append(d.fn.clone())
    ws = torch.zeros(max(d._ws.numel() for d in decs), dtype=torch.uint8, device=cuda)
    for i in (0, 0, 0, 0, 1, 1, 0, 2, 2, 2, 1, 0):
        d = decs[i]
        d._step_plan()
        d._plan.ws = ptr(ws)
        d.fn.fill_(7.0)
        q.check(q.lib().qlmb_dec_step(d._plan, stream_ptr()))
        assert torch.equal(d.fn, want[i]), i
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("B,D,Tm", [(5, 128, 40), (16, 768, 300), (17, 256, 64), (33, 512, 100), (64, 768, 1024)])
def test_decode_attention_on_the_projections_slice_sums(cuda, B, D, Tm):
    """q, k, v, rotation, append and attention in two launches: the same bits, in output and caches, as the separate entries; a
    slot past its cache is reported and left alone."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import block, qlm
    from cudalm_c_b200._lib import ptr, stream_ptr
    g = torch.Generator(device=cuda); g.manual_seed(B)
    Q = qlm.Qlm([(0, 3 * D * D)], 3 * D * D, cuda)
    Q.init_from(torch.randn(3 * D * D, device=cuda, generator=g) * 0.02, render=False)
    x = torch.randn(B, D, device=cuda, generator=g).bfloat16()
    gamma = torch.rand(D, device=cuda, generator=g) + 0.5
    cosb, sinb = block.rope_tables(Tm, 64, device=cuda)
    pos = torch.randint(0, Tm, (B,), device=cuda, generator=g, dtype=torch.int32)
    pos[0], pos[1] = 0, Tm - 1
    for past in (False, True):
        if past:
            pos[2] = Tm
        c1 = [torch.randn(B, Tm, D, device=cuda, generator=g).bfloat16() for _ in range(2)]
        c2 = [t.clone() for t in c1]
        o1, o2 = (torch.full((B, D), 3.0, device=cuda).bfloat16() for _ in range(2))
        y = torch.empty(3 * B, D, dtype=torch.bfloat16, device=cuda)
        q.check(q.lib().qlmb_dec_qkv(ptr(y), ptr(c1[0]), ptr(c1[1]), ptr(x), ptr(gamma), ptr(Q.d), ptr(Q.s), ptr(cosb), ptr(sinb),
                                     ptr(pos), B, D, 64, Tm, stream_ptr()))
        q.check(q.lib().qlmb_dec_attn(ptr(o1), ptr(y), ptr(c1[0]), ptr(c1[1]), ptr(pos), 0, B, Tm, D // 64, D // 64, 64, stream_ptr()))
        if past:
            assert q.lib().qlmb_check_device(None) == 4
        q.check(q.lib().qlmb_dec_qkv_attn(ptr(o2), ptr(c2[0]), ptr(c2[1]), ptr(x), ptr(gamma), ptr(Q.d), ptr(Q.s), ptr(cosb),
                                          ptr(sinb), ptr(pos), B, D, Tm, stream_ptr()))
        torch.cuda.synchronize()
        if past:
            assert q.lib().qlmb_check_device(None) == 4 and b"error code 201" in q.lib().qlmb_last_error()
        assert torch.equal(o1, o2) and all(torch.equal(a, b) for a, b in zip(c1, c2))
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("N,D,F,E,K", [(5, 256, 256, 8, 2), (9, 128, 384, 4, 1), (33, 768, 512, 32, 2), (64, 768, 1536, 32, 2),
                                       (64, 256, 256, 16, 2), (64, 256, 256, 8, 4)])
def test_output_projection_and_experts_in_one_call(cuda, N, D, F, E, K):
    """wo, residual, norm and the expert layer: the same bits as the two entries, with the slice sums added in the router's launch
    and (4 x 64 routed rows) without."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import moe, qlm
    from cudalm_c_b200._lib import ptr, stream_ptr
    g = torch.Generator(device=cuda); g.manual_seed(N + D)

    def weights(n):
        Q = qlm.Qlm([(0, n)], n, cuda)
        Q.init_from(torch.randn(n, device=cuda, generator=g) * 0.02, render=False)
        return Q.d, Q.s
    wo, w1, w3, w2 = weights(D * D), weights(E * D * F), weights(E * D * F), weights(E * F * D)
    wr = torch.randn(D, E, device=cuda, generator=g) * 0.1
    layer = moe.MoeLayerState(N, D, F, E, K, w1, w3, w2, wr, aux=0.0)
    att, res = (torch.randn(N, D, device=cuda, generator=g).bfloat16() for _ in range(2))
    gamma = torch.rand(D, device=cuda, generator=g) + 0.5
    a, b = ([torch.zeros(N, D, device=cuda).bfloat16() for _ in range(3)] for _ in range(2))
    q.check(q.lib().qlmb_gemv_decode_res_norm(ptr(a[0]), ptr(a[1]), ptr(att), ptr(wo[0]), ptr(wo[1]), ptr(res), ptr(gamma), N, D, D,
                                              stream_ptr()))
    layer.decode(a[0], a[1], out=a[2])
    q.check(q.lib().qlmb_dec_wo_moe(layer.c, layer.arena_ptr, ptr(b[2]), ptr(b[0]), ptr(b[1]), ptr(att), ptr(wo[0]), ptr(wo[1]),
                                    ptr(res), ptr(gamma), stream_ptr()))
    torch.cuda.synchronize()
    assert float(a[2].float().norm()) > 0 and all(torch.equal(x, y) for x, y in zip(a, b))
    q.check(q.lib().qlmb_check_device(None))


@pytest.mark.parametrize("K,counts", [(1, [64] + [0] * 7), (1, [0] * 7 + [33]), (2, [32, 32] + [0] * 6), (2, [16, 17, 0, 1, 15, 33, 46, 0]),
                                      (2, [8] * 16), (2, [64] + [0] * 14 + [64])])
def test_expert_rows_in_groups_of_sixteen(cuda, K, counts):
    """Routings that fill an expert's first group of sixteen rows in part, fully, and several more, and leave experts without
    rows: the experts' contribution alone (no residual) against float64 over the same choices."""
    import cudalm_c_b200 as q
    from cudalm_c_b200 import moe, qlm
    E, D, F = len(counts), 128, 256
    N = sum(counts) // K
    g = torch.Generator(device=cuda); g.manual_seed(E + counts[0])

    def weights(n):
        Q = qlm.Qlm([(0, n)], n, cuda)
        P = torch.randn(n, device=cuda, generator=g) * 0.02
        Q.init_from(P)
        return (Q.d, Q.s), P.double()
    (q1, p1), (q3, p3), (q2, p2) = weights(E * D * F), weights(E * D * F), weights(E * F * D)
    # token n's choices through features that only the router reads: logits 16, and 15.6 for the second one (no count is above
    # N, so that a token's two are different experts)
    slots = [e for e, c in enumerate(counts) for _ in range(c)]
    x = torch.randn(N, D, device=cuda, generator=g) * 0.1
    x[:, :2 * E] = 0.0
    for n in range(N):
        for k in range(K):
            x[n, k * E + slots[n + k * N]] = 4.0 - 0.1 * k
    x = x.bfloat16()
    wr = torch.zeros(D, E, device=cuda)
    wr[torch.arange(E), torch.arange(E)] = 4.0
    wr[E + torch.arange(E), torch.arange(E)] = 4.0
    layer = moe.MoeLayerState(N, D, F, E, K, q1, q3, q2, wr, aux=0.0)
    out = layer.decode(torch.zeros(N, D, device=cuda).bfloat16(), x)
    torch.cuda.synchronize()
    q.check(q.lib().qlmb_check_device(None))
    assign = layer.member("assign", (K, N), torch.int32).long()
    gate = layer.member("gate", (K, N), torch.float32).double()
    assert torch.bincount(assign.flatten(), minlength=E).tolist() == counts
    ref = torch.zeros(N, D, dtype=torch.float64, device=cuda)
    w1, w3, w2 = p1.view(E, D, F), p3.view(E, D, F), p2.view(E, F, D)
    for k in range(K):
        for n in range(N):
            e = int(assign[k, n])
            h = x[n].double()
            gg = h @ w1[e]
            ref[n] += gate[k, n] * ((gg * torch.sigmoid(gg) * (h @ w3[e])) @ w2[e])
    # gate, up, their product, the expert's output and the sum are rounded to bf16, and so may the weights be: six roundings of at
    # most 2^-9 and 2^-9 sqrt(6 / 3) together by their root mean square, times four for the largest of the tokens
    err = (out.double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err.max()) < 4 * 2 ** -9 * 2 ** 0.5, err.tolist()
