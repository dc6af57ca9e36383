"""Kernels whose blocks may start before the one ahead of them ends: back to back, behind another
stream's event and in a captured graph they give the bits that they give one at a time."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _chain(T, D, H, Hk, dh, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + T)
    r = lambda *s, std=1.0: (torch.randn(*s, generator=g, device=DEV) * std).to(torch.bfloat16)
    w = dict(x=r(T, D), norm=r(D) * 0.1 + 1, qkv=r((H + 2 * Hk) * dh, D, std=D ** -0.5), o=r(D, H * dh, std=0.05),
             gu=r(4 * D, D, std=D ** -0.5), down=r(D, 2 * D, std=D ** -0.5), dy=r(T, D, std=0.1),
             pos=torch.arange(T, dtype=torch.int32, device=DEV),
             cu=torch.tensor([0, T // 3, T], dtype=torch.int32, device=DEV))
    nq, nk = H * dh, Hk * dh

    def run(sync):
        done = torch.cuda.synchronize if sync else (lambda: None)
        y, rstd = F.rmsnorm_fwd(w["x"], w["norm"], 1e-6); done()
        qkv = F.gemm(y, w["qkv"]); done()
        F.rope_(qkv, w["pos"], col0=0, heads=H + Hk, dh=dh, rot=dh, theta=1e4); done()
        q, k, v = (t.reshape(T, -1, dh) for t in (qkv[:, :nq], qkv[:, nq:nq + nk], qkv[:, nq + nk:]))
        out, lse = F.attention_varlen(q, k, v, w["cu"], T); done()
        h = F.gemm(out.reshape(T, nq), w["o"]); done()
        gu = F.gemm(h, w["gu"]); done()
        a = F.swiglu_fwd(gu); done()
        z = F.gemm(a, w["down"]); done()
        da = F.gemm(w["dy"], w["down"], b_mn=True); done()
        dgu = F.swiglu_bwd(gu, da); done()
        grads = F.attention_varlen_bwd(q, k, v, out, lse, out, w["cu"], T); done()
        return y, rstd, qkv, out, lse, h, a, z, dgu, *grads
    return w, run


SHAPES = [(7, 128, 2, 1, 64), (300, 256, 4, 2, 64), (1999, 1024, 8, 2, 128), (6000, 512, 4, 1, 256)]


@pytest.mark.parametrize("shape", SHAPES)
def test_back_to_back_calls_have_the_bits_of_single_ones(shape):
    _, run = _chain(*shape)
    want = run(True)
    runs = [run(False) for _ in range(12)]
    torch.cuda.synchronize()
    _lib.check_status()
    assert all(torch.equal(a, b) for got in runs for a, b in zip(got, want))


@pytest.mark.parametrize("shape", SHAPES[:3])
def test_captured_calls_have_the_bits_of_single_ones(shape):
    _, run = _chain(*shape)
    want = run(True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = run(False)
    for _ in range(3):
        for t in got:
            t.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_a_wait_for_another_stream_holds():
    w, run = _chain(*SHAPES[2])
    x, side = w["x"].clone(), torch.cuda.Stream()
    want = run(True)
    for _ in range(6):
        run(False)                                     # the kernel ahead of the wait is a chained one
        w["x"].zero_()
        ready = torch.cuda.Event()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(20):
                torch.empty(1 << 24, device=DEV).fill_(1.0)
            w["x"].copy_(x)
            ready.record()
        F.rmsnorm_fwd(w["dy"], w["norm"], 1e-6)        # so that the wait lies between two chained kernels
        torch.cuda.current_stream().wait_event(ready)
        got = run(False)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want))
