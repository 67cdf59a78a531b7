"""Which operators a decode step's chain calls, by the shape: the calls are recorded, nothing is launched, so no GPU is needed."""
import types

import pytest
import torch

from cudalm_c_b200 import block, model
from cudalm_c_b200._lib import QlmbError, check


class Recorder:
    """Stands for the library: notes the name of every call; the cached attention answers as the library does."""

    def __init__(self):
        self.names = []

    def __getattr__(self, name):
        def call(*args):
            self.names.append(name)
            return int(name == "qlmb_dec_attn" and args[10] != 64)
        return call


def decoder(B, H, hd, KV):
    cfg = model.Config(L=1, D=H * hd, H=H, KV=KV, hd=hd, E=4, K=2, F=128, V=256, T=64, B=1)
    t = torch.zeros(1)
    d = object.__new__(model.Decoder)
    d.m = types.SimpleNamespace(c=cfg, dev="cpu", emb=t, nf=t, fl=[dict(an1=t, an2=t)], layers=[dict(w={k: (t, t) for k in ("wq", "wk", "wv", "wo")})])
    d.B, d.Tm, d.tok, d.pos, d.cosb, d.sinb, d.K, d.V = B, 64, t, t, t, t, [t], [t]
    d.moes = [types.SimpleNamespace(c=None, arena_ptr=0, decode=lambda a, b: a)]
    return d


@pytest.mark.parametrize("B", [1, 4, 5, 8, 64])
@pytest.mark.parametrize("hd", [32, 128])
def test_other_head_dimensions_stay_refused(monkeypatch, B, hd):
    """The attention has heads of 64 only; the operator that joins it with the projections must not take a model with others for
    one with D / 64 heads."""
    monkeypatch.setattr(block, "embed", lambda *a, **k: torch.zeros(1))
    L = Recorder()
    with pytest.raises(QlmbError):
        decoder(B, 256 // hd, hd, 256 // hd)._chain(L, check, lambda t: 0, lambda: 0)
    assert L.names == ["qlmb_dec_qkv", "qlmb_dec_attn"]


@pytest.mark.parametrize("B,joined", [(4, False), (5, True), (64, True)])
def test_heads_of_64_with_many_slots_join_projections_and_attention(monkeypatch, B, joined):
    monkeypatch.setattr(block, "embed", lambda *a, **k: torch.zeros(1))
    monkeypatch.setattr(block, "rmsnorm_fwd", lambda *a, **k: (torch.zeros(1), None))
    L = Recorder()
    decoder(B, 4, 64, 4)._chain(L, check, lambda t: 0, lambda: 0)
    assert L.names == (["qlmb_dec_qkv_attn", "qlmb_dec_wo_moe"] if joined else ["qlmb_dec_qkv", "qlmb_dec_attn", "qlmb_gemv_decode_res_norm"])
