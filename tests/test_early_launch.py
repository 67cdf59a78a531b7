"""Kernels that start before the kernel in front of them has ended (programmatic dependent launches).

What they read may be what that kernel writes: an optimizer step directly in front of a decode step writes the router
matrix, the codes and the scales.  On the CPU the sources are held to the rule (nothing is loaded ahead of the wait); on
the GPU results behind a writer equal those behind a synchronisation."""
import os
import re

import pytest
import torch

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudalm_c_b200", "csrc")
# a global load: the intrinsics, the library's own load helpers, a load lambda of a kernel
LOAD = re.compile(r"__ld\w+\s*\(|\bld_\w+\s*\(|\bfetch\s*\(")


def braces(src, i):
    """The end of the block that opens at src[i]."""
    depth, j = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(src[j], 0)
        j += 1
    return j


def kernels(whole=False):
    """(name, body without comments and, unless `whole`, without the bodies of its lambdas) of every __global__ function."""
    out = []
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as h:
            src = re.sub(r"//[^\n]*", "", h.read())
        for m in re.finditer(r"__global__\s+void\b", src):
            i = src.index("{", m.end())
            name = re.findall(r"(\bk_\w+)\s*\(", src[m.end():i])[0]
            body = src[i:braces(src, i)]
            while not whole:
                lam = re.search(r"auto \w+ = \[[&=]?\]\s*\([^)]*\)\s*\{", body)
                if not lam:
                    break
                body = body[:lam.start()] + body[braces(body, lam.end() - 1):]
            out.append((name, body))
    return out


def test_nothing_is_loaded_ahead_of_the_wait():
    """In every kernel that can start early the first pdl_wait() stands in front of its first load, and only the name of a
    launch without a writer of weights in front (QUIET, AHEAD) may make it conditional."""
    seen = 0
    for name, body in kernels():
        if "pdl_wait()" not in body:
            continue
        seen += 1
        head = body[:body.index("pdl_wait()")]
        assert not LOAD.search(head), name
        cond = re.findall(r"if \(([^;{}]*)\)\s*(?:\{[^{}]*)?$", head)
        assert not cond or cond[0] in ("quiet != QUIET", "!AHEAD") or name.startswith("k_attn"), (name, cond)
    assert seen > 30


def test_no_early_kernel_promises_read_only_data():
    """__ldg states that nothing writes the data while the kernel runs: not so beside a predecessor that still runs."""
    for name, body in kernels(whole=True):
        assert "pdl_wait()" not in body or "__ldg(" not in body, name


def test_launches_of_few_long_blocks_do_not_start_early():
    """Placed beside the last blocks of their predecessor they would share SMs while others idle."""
    src = {f: open(os.path.join(CSRC, f)).read() for f in ("qlmb_dispatch.cu", "qlmb_block.cu")}
    assert len(re.findall(r"pdl_launch\(false, k_router_logits_tile<[01]>", src["qlmb_dispatch.cu"])) == 2
    assert "pdl_launch(false, k_rmsnorm_bwd," in src["qlmb_block.cu"]


@pytest.mark.gpu
@pytest.mark.parametrize("N", [5, 8, 64])
def test_adamw_on_the_router_directly_before_a_decode_step(cuda, N):
    """qlmb_adamw lets the next kernel start early and writes the router matrix that the next kernel multiplies with."""
    from cudalm_c_b200 import moe, qlm
    D, F, E, K = 1024, 128, 32, 2
    g = torch.Generator(device=cuda); g.manual_seed(N)
    q = []
    for _ in range(3):
        Q = qlm.Qlm([(0, E * D * F)], E * D * F, cuda)
        Q.init_from(torch.randn(E * D * F, device=cuda, generator=g) * 0.02, render=False)
        q.append(Q)
    x, xn = (torch.randn(N, D, device=cuda, generator=g).bfloat16() for _ in range(2))
    G = torch.randn(D * E, device=cuda, generator=g)
    wr0 = torch.randn(D * E, device=cuda, generator=g) * 0.02

    def steps(sync):
        wr = wr0.clone()
        M, V = (torch.zeros(D * E, dtype=torch.int16, device=cuda) for _ in range(2))
        layer = moe.MoeLayerState(N, D, F, E, K, *((a.d, a.s) for a in q), wr.view(D, E), aux=0.0)
        outs = []
        for t in range(1, 9):
            qlm.adamw(wr, G if t % 2 else -G, M, V, 0.05, 0.9, 0.95, 0.0, 1.0, 1.0)
            if sync:
                torch.cuda.synchronize()
            layer.decode(x, xn)
            outs.append(layer.member("rt", (N, E), torch.float32).clone())
        return torch.stack(outs)
    want = steps(True)
    assert not torch.equal(want[0], want[1])
    for _ in range(20):
        assert torch.equal(steps(False), want)


@pytest.mark.gpu
@pytest.mark.parametrize("B", [1, 2, 4, 8, 33])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_optimizer_step_directly_before_a_gemv(cuda, B, layout):
    """The codes and scales that a GEMV multiplies with are those of the optimizer step in front of it."""
    from cudalm_c_b200 import _lib, linear, qlm
    K, N = 1024, 8192
    g = torch.Generator(device=cuda); g.manual_seed(B)
    w = torch.randn(K * N, device=cuda, generator=g) * 0.02
    G = torch.randn(K * N, device=cuda, generator=g)
    for dt in (torch.bfloat16, torch.float32):
        x = torch.randn(B, K, device=cuda, generator=g).to(dt)

        def steps(sync):
            Q = qlm.Qlm([(0, K * N)], K * N, cuda)
            Q.init_from(w, render=False)
            outs = []
            for t in range(1, 7):
                Q.step(None, G if t % 2 else -G, 0.05, 0.9, 0.95, 0.1, t)
                if sync:
                    torch.cuda.synchronize()
                outs.append(linear.gemv_decode(x, Q.d, Q.s, getattr(_lib, layout), N))
            return torch.stack(outs)
        want = steps(True)
        assert not torch.equal(want[0], want[1])
        for _ in range(4):
            assert torch.equal(steps(False), want)
