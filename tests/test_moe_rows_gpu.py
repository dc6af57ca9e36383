"""Sorted expert rows: layout and its inverse, padding, the activation's backward and the router's
gradient, from one token to many blocks, with idle and crowded experts."""
import pytest
import torch
import torch.nn.functional as TF

from shadowspill_b200.ops import _lib, moe

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [(1, 1, 1), (1, 8, 2), (33, 8, 8), (700, 64, 8), (513, 65, 3), (300, 128, 8), (90, 512, 32), (5000, 16, 4)]


def _route(T, E, k, renorm, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + T)
    logits = torch.randn(T, E, generator=g, device=DEV) + 3.0 * torch.randn(1, E, generator=g, device=DEV)
    return g, logits, *moe.route(logits, k, renorm)


@pytest.mark.parametrize("T,E,k", SHAPES)
def test_layout_gather_and_activation(T, E, k):
    g, logits, ids, wts, counts = _route(T, E, k, False)
    assert torch.equal(counts.long(), torch.bincount(ids.reshape(-1).long(), minlength=E))
    lay = moe.Layout(ids, counts)
    off, dest, src = lay.offsets.tolist(), lay.dest.long(), lay.src.long()
    used = off[-1]
    assert off[0] == 0 and [b - a for a, b in zip(off, off[1:])] == [-(-n // 128) * 128 for n in counts.tolist()]
    assert torch.equal(src[dest], torch.arange(T * k, device=DEV)) and int((src >= 0).sum()) == T * k
    start = lay.offsets.long()[ids.reshape(-1).long()]
    assert bool(((dest >= start) & (dest < start + counts.long()[ids.reshape(-1).long()])).all())
    x = torch.randn(T, 72, generator=g, device=DEV).to(torch.bfloat16)
    xs = lay.gather(x)[:used]
    real = src[:used] >= 0
    assert torch.equal(xs[real], x[src[:used][real] // k]) and not bool(xs[~real].any())
    # activation backward against autograd in fp64 on the same bf16 inputs
    Fw = 136
    gu = torch.zeros(lay.rows, 2 * Fw, dtype=torch.bfloat16, device=DEV)
    d = torch.zeros(lay.rows, Fw, dtype=torch.bfloat16, device=DEV)
    rows = dest
    gu[rows] = torch.randn(T * k, 2 * Fw, generator=g, device=DEV).to(torch.bfloat16)
    d[rows] = torch.randn(T * k, Fw, generator=g, device=DEV).to(torch.bfloat16)
    h = lay.swiglu(gu)
    dgu, hw, dots = lay.act_bwd(gu, d, wts)
    _lib.check_status()
    leaf = gu[rows].double().requires_grad_(True)
    href = TF.silu(leaf[:, :Fw]) * leaf[:, Fw:]
    w = wts.double().reshape(-1, 1)
    (want,) = torch.autograd.grad(href, leaf, w * d[rows].double())
    rel = lambda a, b: float((a.double() - b).norm() / (b.norm() + 1e-30))
    # silu and h are rounded to bf16 (2^-9 each), the results once more
    assert rel(h[rows], href.detach()) < 8e-3 and rel(dgu[rows], want) < 8e-3
    assert rel(hw[rows], w * href.detach()) < 8e-3
    assert rel(dots.reshape(-1), (d[rows].double() * h[rows].double()).sum(1)) < 1e-5
    pad = torch.nonzero(~real).reshape(-1)
    assert not bool(dgu[pad].any()) and not bool(hw[pad].any())


@pytest.mark.parametrize("T,E,k", SHAPES)
@pytest.mark.parametrize("renorm", [True, False])
def test_router_gradient(T, E, k, renorm):
    g, logits, ids, wts, _ = _route(T, E, k, renorm, seed=3)
    dwts = torch.randn(T, k, generator=g, device=DEV)
    got = moe.route_bwd(logits, ids, wts, dwts, renorm)
    leaf = logits.double().requires_grad_(True)
    moe._weights_from_logits(leaf, ids.long(), renorm).backward(dwts.double())
    # fp32 weights and sums; for one expert or one pick the exact gradient may be zero
    assert float((got.double() - leaf.grad).abs().max()) < 1e-5 * (1.0 + float(leaf.grad.abs().max()))


@pytest.mark.parametrize("M,N", [(256, 512), (136, 72)])
def test_bank_gradient_leaves_out_blocks_of_padding(M, N):
    loads = [0, 1, 63, 64, 65, 127, 128, 129, 192, 300, 0]
    ids = torch.repeat_interleave(torch.arange(len(loads), dtype=torch.int32, device=DEV),
                                  torch.tensor(loads, device=DEV)).reshape(-1, 1)
    lay = moe.Layout(ids, torch.tensor(loads, dtype=torch.int32, device=DEV))
    g = torch.Generator(device=DEV).manual_seed(M)
    dy, x = (lay.gather(torch.randn(ids.numel(), w, generator=g, device=DEV).to(torch.bfloat16)) for w in (M, N))
    out = torch.full((len(loads), M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    moe.grouped_wgrad(dy, x, lay, out, False)
    whole, lay.counts = torch.full_like(out, 5.0), None            # the padding contracted as well
    moe.grouped_wgrad(dy, x, lay, whole, False)
    _lib.check_status()
    assert torch.equal(out, whole)
    off = lay.offsets.tolist()
    for e, n in enumerate(loads):
        want = dy[off[e]:off[e] + n].double().T @ x[off[e]:off[e] + n].double()
        # fp32 sums of exact products, rounded to bf16 once (2^-9 of each value)
        assert float((out[e].double() - want).abs().max()) <= 2.0 ** -8 * (1e-3 + float(want.abs().max() if n else 0))


@pytest.mark.parametrize("E,k,finite", [(4, 3, 2), (8, 8, 1), (64, 8, 3), (65, 6, 0), (512, 32, 31)])
@pytest.mark.parametrize("renorm", [True, False])
def test_fewer_comparable_scores_than_picks(E, k, finite, renorm):
    """Masked experts (scores of -inf) fill up the picks: each once, with no weight and no gradient of their own."""
    T = 300
    g = torch.Generator(device=DEV).manual_seed(E + k)
    logits = torch.full((T, E), -float("inf"), device=DEV)
    open_ = torch.rand(T, E, generator=g, device=DEV).argsort(1)[:, :finite]
    logits.scatter_(1, open_, torch.randn(T, finite, generator=g, device=DEV))
    ids, wts, counts = moe.route(logits, k, renorm)
    assert int(ids.min()) >= 0 and int(ids.max()) < E
    assert bool((ids.sort(1).values.diff(dim=1) > 0).all())                # no expert twice
    assert torch.equal(counts.long(), torch.bincount(ids.reshape(-1).long(), minlength=E))
    if finite == 0:
        return                                                             # no weights to speak of: 0 / 0
    assert torch.equal(ids[:, :finite].long(), logits.topk(finite, 1).indices)
    leaf = logits.double().requires_grad_(True)
    want = (leaf.gather(1, ids.long()).softmax(1) if renorm else leaf.softmax(1).gather(1, ids.long()))
    assert float((wts.double() - want).abs().max()) < 1e-6
    dwts = torch.randn(T, k, generator=g, device=DEV)
    want.backward(dwts.double())
    got = moe.route_bwd(logits, ids, wts, dwts, renorm)
    assert bool(torch.isfinite(got).all())
    # fp32 products and sums of up to 32 terms of order one
    assert float((got.double() - leaf.grad).abs().max()) < 1e-5


def _off_by_8_bytes(*shape):
    n = 1
    for d in shape:
        n *= d
    return torch.zeros(n + 4, dtype=torch.bfloat16, device=DEV)[4:].view(*shape)


@pytest.mark.parametrize("accumulate", [False, True])
def test_grouped_outputs_on_8_byte_boundaries(accumulate):
    """The staged stores take them (TMA would not); experts without rows among them. On 2 bytes they are refused."""
    E, T, D, N, k = 8, 300, 136, 200, 2
    g = torch.Generator(device=DEV).manual_seed(3)
    logits = torch.randn(T, E, generator=g, device=DEV)
    logits[:, 5] = -1e4
    ids, _, counts = moe.route(logits, k, True)
    assert int(counts[5]) == 0
    lay = moe.Layout(ids, counts)
    used = int(lay.used)
    x = torch.randn(T, D, generator=g, device=DEV).bfloat16()
    bank = (torch.randn(E, N, D, generator=g, device=DEV) * 0.1).bfloat16()
    xs = lay.gather(x)
    want = moe.grouped_linear(xs, bank, lay)
    got = moe.grouped_linear(xs, bank, lay, out=_off_by_8_bytes(lay.rows, N))
    assert got.data_ptr() % 16 == 8 and torch.equal(got[:used], want[:used])
    start = torch.randn(E, N, D, generator=g, device=DEV).bfloat16()
    a, b = start.clone(), _off_by_8_bytes(E, N, D).copy_(start)
    moe.grouped_wgrad(want, xs, lay, a, accumulate)
    moe.grouped_wgrad(want, xs, lay, b, accumulate)
    assert b.data_ptr() % 16 == 8 and torch.equal(a, b)
    assert accumulate or not bool(b[5].any())
    flat = torch.zeros(lay.rows * N + 1, dtype=torch.bfloat16, device=DEV)[1:].view(lay.rows, N)
    with pytest.raises(RuntimeError):
        moe.grouped_linear(xs, bank, lay, out=flat)
    torch.cuda.synchronize()
    _lib.check_status()
