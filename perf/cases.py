"""What this framework is timed on: the work its users have it do, through its public entry points.

A case is one of seven calls, by its "op":

  gemv     linear.gemv_decode: a few decode rows times 4-bit matrices
  linear   linear.linear_fwd + linear_dgrad + linear_wgrad: one quantised linear of a training step
  moe      moe.MoeLayerState.forward (+ .backward): one layer of routed expert FFNs on 4-bit weights
  attn     attn.attn_fwd + attn.attn_bwd: causal attention, heads of 64
  update   qlm.gnorm + Qlm.step + qlm.adamw on the float spans: clip and integer AdamW, as QlmModel.update does it
  decode   model.Decoder.step: one token for every live slot, replayed from a CUDA graph as a serving loop does
  train    model.QlmModel.forward + .backward: a training step up to its gradients

Inputs are synthetic with the distributions the path meets in training from random initialisation: activations
N(0, 1), weights N(0, 0.02) quantised by the library itself, gradients N(0, 1e-3), token ids uniform.
"""
import math

import torch

from cudalm_c_b200 import attn, linear, model, moe, qlm
from cudalm_c_b200._lib import KN, NK

BYTES_PER_WEIGHT = 0.5 + 4.0 / 128          # a 4-bit code and its share of the group's fp32 scale
DTYPES = {"bf16": (torch.bfloat16, 2), "f32": (torch.float32, 4)}
LAYOUTS = {"KN": KN, "NK": NK}

# The ~120 M-active-parameter MoE language model that this repository trains and decodes.
LM = dict(L=12, D=768, H=12, E=32, K=2, F=1536, V=16384)


def listed():
    return [
        # one attention projection of one decode slot: the smallest call, all launch and host latency
        dict(name="gemv_1x768x768", op="gemv", B=1, K=768, N=768, mats=1, layout="KN", dtype="bf16"),
        # four large matrices one after the other for one slot: the weight stream itself
        dict(name="gemv_1x4096x16384", op="gemv", B=1, K=4096, N=16384, mats=4, layout="KN", dtype="bf16"),
        # generation for one user, a small batch and a full server (prompts of 128, in the middle of 256 new tokens)
        dict(name="decode_b1", op="decode", B=1, fill=256, Tm=1024, **LM),
        dict(name="decode_b8", op="decode", B=8, fill=256, Tm=1024, **LM),
        dict(name="decode_b64", op="decode", B=64, fill=256, Tm=1024, **LM),
        # a dense quantised linear with fp32 activations, [out, in] weights
        dict(name="linear_8192x512x2048_f32", op="linear", M=8192, K=512, N=2048, layout="NK", dtype="f32"),
        # a model-width projection on a ragged number of rows, bf16 activations, [in, out] weights
        dict(name="linear_1003x768x768_bf16", op="linear", M=1003, K=768, N=768, layout="KN", dtype="bf16"),
        # the expert layer of a training step
        dict(name="moe_train_8192", op="moe", N=8192, D=768, F=1536, E=32, K=2, backward=True),
        # the expert layer of a prompt: forward only, ragged
        dict(name="moe_prefill_333", op="moe", N=333, D=768, F=1536, E=32, K=2, backward=False),
        # the attention of a training step
        dict(name="attn_8x1024x12", op="attn", B=8, T=1024, H=12, KV=12, win=0),
        # the optimizer over a flat set of 4-bit weights
        dict(name="update_126m", op="update", n=125829120, spans=1, floats=0),
        # the whole model: 8 sequences of 1024 tokens, forward, head and backward
        dict(name="train_8x1024", op="train", B=8, T=1024, **LM),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _wide(rng, lo, hi):
    """A matrix dimension: a multiple of the 128 weights that share a scale."""
    return 128 * _log(rng, lo // 128, hi // 128)


def draw(rng):
    op = rng.choice(("gemv", "decode", "decode", "linear", "moe", "attn", "update", "train"))
    if op == "gemv":
        return dict(op=op, B=_log(rng, 1, 64), K=_wide(rng, 512, 4096), N=_wide(rng, 512, 16384), mats=rng.randint(1, 4),
                    layout=rng.choice(("KN", "KN", "NK")), dtype=rng.choice(("bf16", "bf16", "bf16", "f32")))
    if op == "linear":
        return dict(op=op, M=_log(rng, 65, 8192), K=_wide(rng, 256, 2048), N=_wide(rng, 256, 2048),
                    layout=rng.choice(("KN", "NK")), dtype=rng.choice(("bf16", "f32")))
    if op == "moe":
        return dict(op=op, N=_log(rng, 65, 8192), D=_wide(rng, 256, 1024), F=_wide(rng, 256, 2048),
                    E=rng.choice((4, 8, 16, 32)), K=rng.choice((1, 2, 2)), backward=rng.random() < 0.6)
    if op == "attn":
        h = rng.choice((4, 8, 12, 16))
        t = _log(rng, 64, 2048)
        return dict(op=op, B=max(1, min(8, 8192 // t, rng.randint(1, 8))), T=t, H=h, KV=rng.choice((h, h, h // 2, h // 4)),
                    win=rng.choice((0, 0, 0, 256)))
    if op == "update":
        return dict(op=op, n=2 * _log(rng, 50000, 60000000), spans=rng.randint(1, 12), floats=rng.choice((0, 1000, 20001)))
    h = rng.choice((4, 8, 12, 16))
    m = dict(L=rng.randint(1, 12), D=64 * h, H=h, E=rng.choice((8, 16, 32)), K=rng.choice((1, 2, 2)), F=_wide(rng, 256, 1536),
             V=256 * rng.randint(16, 64))
    if op == "decode":
        fill = _log(rng, 16, 512)
        return dict(op=op, B=_log(rng, 1, 64), fill=fill, Tm=rng.choice((640, 1024)), **m)
    m["L"] = rng.randint(1, 4)
    return dict(op=op, B=rng.randint(1, 8), T=_log(rng, 64, 1024), **m)


def _quantised(count, g, dev):
    """`count` weights N(0, 0.02) as 4-bit codes and group scales."""
    w = torch.randn(count, device=dev, generator=g) * 0.02
    q = qlm.Qlm([(0, count)], count, dev)
    q.init_from(w, render=False)
    return q


def _model(c, B, T, g, dev, aux):
    """A model with its parameters as a checkpoint holds them: one flat fp32 vector."""
    cfg = model.Config(L=c["L"], D=c["D"], H=c["H"], KV=c["H"], hd=64, E=c["E"], K=c["K"], F=c["F"], V=c["V"], T=T, B=B)
    o = model.Offsets(cfg)
    p = torch.randn(o.total, device=dev, generator=g) * 0.02
    for lo in o.layers:
        for nm in ("wo", "w2"):
            a, n = lo[nm]
            p[a:a + n] /= math.sqrt(2.0 * cfg.L)
        for nm in ("an1", "an2"):
            a, n = lo[nm]
            p[a:a + n] = 1.0
    p[o.nf:o.nf + cfg.D] = 1.0
    return model.QlmModel(cfg, dev, aux=aux, P_init=p)


def _positions(c, seed):
    """Every slot's position of a decode step: slots joined at different times."""
    g = torch.Generator()
    g.manual_seed(seed)
    return torch.randint((c["fill"] + 1) // 2, c["fill"] + 1, (c["B"],), generator=g, dtype=torch.int32)


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    c, op = case, case["op"]
    s = dict(c)

    def acts(rows, cols, dt=torch.bfloat16):
        return torch.randn(rows, cols, device=dev, generator=g).to(dt)

    if op == "gemv":
        s["q"] = [_quantised(c["K"] * c["N"], g, dev) for _ in range(c["mats"])]
        s["x"] = acts(c["B"], c["K"], DTYPES[c["dtype"]][0])
    elif op == "linear":
        s["q"] = _quantised(c["K"] * c["N"], g, dev)
        s["x"], s["dy"] = (acts(c["M"], n, DTYPES[c["dtype"]][0]) for n in (c["K"], c["N"]))
        s["dw"] = torch.zeros(c["K"] * c["N"], device=dev)
    elif op == "moe":
        n, d, f, e = c["N"], c["D"], c["F"], c["E"]
        q1, q3, q2 = (_quantised(e * d * f, g, dev) for _ in range(3))
        s["wr"] = torch.randn(d, e, device=dev, generator=g) * 0.02
        s["layer"] = moe.MoeLayerState(n, d, f, e, c["K"], (q1.d, q1.s), (q3.d, q3.s), (q2.d, q2.s), s["wr"], aux=0.03)
        s["q"] = (q1, q3, q2)
        s["fi"], s["fn"] = acts(n, d), acts(n, d)
        if c["backward"]:
            s["dout"] = acts(n, d)
            s["dw"] = [torch.zeros(e, d, f, device=dev), torch.zeros(e, d, f, device=dev), torch.zeros(e, f, d, device=dev),
                       torch.zeros(d, e, device=dev)]
    elif op == "attn":
        rows = c["B"] * c["T"]
        s["q"], s["k"], s["v"], s["da"] = (acts(rows, 64 * h) for h in (c["H"], c["KV"], c["KV"], c["H"]))
    elif op == "update":
        # spans of unequal length, each followed by a float span (gains, router, embedding) when there are any
        per = c["n"] // c["spans"] // 2 * 2
        mats, off = [], 0
        for i in range(c["spans"]):
            m = per - 2 * (i * 37 % 64) if c["spans"] > 1 else c["n"]
            mats.append((off, m))
            off += m + c["floats"]
        p = torch.randn(off, device=dev, generator=g) * 0.02
        s["g"] = torch.randn(off, device=dev, generator=g) * 1e-3
        s["q"] = qlm.Qlm(mats, off, dev)
        s["q"].init_from(p, render=False)
        s["fp"] = [p[a:a + m].clone() for a, m, _ in s["q"].fs]
        s["gs"] = torch.ones(2, device=dev)
        s["t"] = 0
    elif op == "decode":
        m = _model(c, 1, max(c["fill"], 64), g, dev, 0.0)
        d = model.Decoder(m, c["B"], c["Tm"])
        d.prefill(torch.randint(0, c["V"], (c["B"], c["fill"]), device=dev, generator=g, dtype=torch.int32))
        s["first"] = d.tok.clone()
        s["pos"] = _positions(c, seed).repeat(2).to(dev)

        def step():
            # the slots as the scheduler left them, then their next token
            d.pos2.copy_(s["pos"])
            d.tok.copy_(s["first"])
            d.step()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
            step()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            step()
        s["dec"], s["model"] = d, m
    elif op == "train":
        n = c["B"] * c["T"]
        s["model"] = _model(c, c["B"], c["T"], g, dev, 0.03)
        s["tok"], s["tgt"] = (torch.randint(0, c["V"], (n,), device=dev, generator=g, dtype=torch.int32) for _ in range(2))
    else:
        raise ValueError(op)
    return s


def run(s):
    op = s["op"]
    if op == "gemv":
        return [linear.gemv_decode(s["x"], q.d, q.s, LAYOUTS[s["layout"]], s["N"]) for q in s["q"]]
    if op == "linear":
        q, lay = s["q"], LAYOUTS[s["layout"]]
        y = linear.linear_fwd(s["x"], q.d, q.s, lay, s["N"])
        dx = linear.linear_dgrad(s["dy"], q.d, q.s, lay, s["K"])
        dw = linear.linear_wgrad(s["dw"], s["dy"], s["x"], lay, beta=0.0)
        return dict(y=y, dx=dx, dw=dw)
    if op == "moe":
        out = s["layer"].forward(s["fi"], s["fn"])
        if not s["backward"]:
            return dict(out=out)
        dfn = s["layer"].backward(s["dout"], s["fn"], *s["dw"], beta=0.0)
        return dict(out=out, dfn=dfn, dw=s["dw"])
    if op == "attn":
        o, lse = attn.attn_fwd(s["q"], s["k"], s["v"], s["B"], s["T"], s["H"], s["KV"], s["win"])
        dq, dk, dv, _ = attn.attn_bwd(s["q"], s["k"], s["v"], o, s["da"], lse, s["B"], s["T"], s["H"], s["KV"], s["win"])
        return dict(o=o, lse=lse, dq=dq, dk=dk, dv=dv)
    if op == "update":
        q = s["q"]
        s["t"] += 1
        qlm.gnorm(s["g"], out=s["gs"])
        q.step(None, s["g"], 3e-4, 0.9, 0.95, 0.1, s["t"], gscale=1.0, gsp=s["gs"])
        bc1, bc2 = qlm.bias_corrections(0.9, 0.95, s["t"])
        for (off, n, cs), p in zip(q.fs, s["fp"]):
            qlm.adamw(p, s["g"][off:off + n], q.Mc[cs:cs + n], q.Vc[cs:cs + n], 3e-4, 0.9, 0.95, 0.0, bc1, bc2, s["gs"])
        if s["t"] % q.servo_every == 0:
            q.servo()
        return dict(gs=s["gs"], d=q.d, r=q.r, m8=q.m8, v8=q.v8, s=q.s, m8s=q.m8s, v8s=q.v8s, Mc=q.Mc, Vc=q.Vc, fp=s["fp"])
    if op == "decode":
        s["graph"].replay()
        d = s["dec"]
        return dict(logits=d.logits, lp=d.olp, k=d.K[-1], v=d.V[-1])
    if op == "train":
        m = s["model"]
        m.forward(s["tok"])
        loss = m.backward(s["tok"], s["tgt"])
        return dict(loss=loss, grad=m.G)
    raise ValueError(op)


def _layer_matmul(c):
    """Weights of one layer that a token is multiplied with: attention, router, its K experts."""
    return 4 * c["D"] * c["D"] + c["D"] * c["E"] + c["K"] * 3 * c["D"] * c["F"]


def _pairs(T, win):
    """(query, key) pairs inside the causal mask of one sequence and head."""
    return T * (T + 1) // 2 if win <= 0 or win >= T else win * (win + 1) // 2 + (T - win) * win


def work(case):
    c, op = case, case["op"]
    if op == "gemv":
        k, n, e = c["K"], c["N"], DTYPES[c["dtype"]][1]
        return dict(bytes=c["mats"] * (k * n * BYTES_PER_WEIGHT + c["B"] * n * e) + c["B"] * k * e, flops=2.0 * c["mats"] * c["B"] * k * n)
    if op == "linear":
        m, k, n, e = c["M"], c["K"], c["N"], DTYPES[c["dtype"]][1]
        return dict(bytes=2 * m * (k + n) * e + k * n * (BYTES_PER_WEIGHT + 4), flops=6.0 * m * k * n)
    if op == "moe":
        n, d, f, e = c["N"], c["D"], c["F"], c["E"]
        w = 3 * d * f
        hit = e * (1.0 - (1.0 - c["K"] / e) ** n)
        back = c["backward"]
        return dict(bytes=hit * w * BYTES_PER_WEIGHT + (5 if back else 3) * n * d * 2 + (e * w * 4.0 if back else 0.0) + d * e * 4,
                    flops=(3 if back else 1) * 2.0 * n * (c["K"] * w + d * e))
    if op == "attn":
        pairs = c["B"] * c["H"] * _pairs(c["T"], c["win"])
        rows = c["B"] * c["T"] * 64 * 2
        return dict(bytes=rows * (4 * c["H"] + 4 * c["KV"]) + c["B"] * c["H"] * c["T"] * 4, flops=7 * 2.0 * pairs * 64)
    if op == "update":
        fl = c["spans"] * c["floats"]
        # gradient 4, digits 0.5 + residual 1 + moments 2 read and written, three scales a group read and written;
        # a float parameter: gradient, value and two bf16 moments
        return dict(bytes=c["n"] * (4 + 2 * 3.5 + 2 * 12 / 128.0) + fl * (4 + 2 * 8), flops=0.0)
    if op == "decode":
        e, b = c["E"], c["B"]
        hit = e * (1.0 - (1.0 - c["K"] / e) ** b)
        w = 4 * c["D"] * c["D"] + hit * 3 * c["D"] * c["F"]
        kv = b * 0.75 * c["fill"] * c["D"] * 2 * 2
        return dict(bytes=c["L"] * (w * BYTES_PER_WEIGHT + c["D"] * e * 4 + kv) + c["V"] * c["D"] * 2 + b * c["V"] * 4,
                    flops=2.0 * b * (c["L"] * _layer_matmul(c) + c["V"] * c["D"]))
    if op == "train":
        n = c["B"] * c["T"]
        stored = c["L"] * (4 * c["D"] * c["D"] + c["E"] * 3 * c["D"] * c["F"])
        return dict(bytes=stored * (BYTES_PER_WEIGHT + 4.0) + c["V"] * c["D"] * 8.0 + n * 12.0,
                    flops=6.0 * n * (c["L"] * _layer_matmul(c) + c["V"] * c["D"])
                    + c["L"] * c["B"] * c["H"] * 7 * 2.0 * _pairs(c["T"], 0) * 64)
    raise ValueError(op)


def tolerance(case):
    op = case["op"]
    if op == "update":
        return "exact"                      # the integer state is defined bit for bit
    if op == "gemv":
        # fp32 rows: fp32 sums of dequantised weights; bf16 rows may be multiplied by bf16(digit * scale)
        return {"rel": 1e-4} if case["dtype"] == "f32" else {"rel": 1e-2}
    if op == "train":
        # Another summation order moves bf16 activations by a rounding here and there, and with them the choice between
        # two experts whose router logits nearly tie (about one choice in a hundred after a few layers, and such a
        # choice moves single gradient elements by their own size).
        return {"rel": 2e-2, "max": 0.99}
    if op == "decode":
        return {"rel": 2e-2, "max": 0.99}   # the same near-ties, for a few of the slots
    return {"rel": 1e-2}                    # bf16 operands, fp32 sums (also behind fp32 inputs and outputs)
