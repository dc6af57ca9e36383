"""The attention kernels at the edges of their tiles: sequences one row short of, at and past 128 and
256 rows, more sequences than a warp has lanes, strided operands and a negative scale."""
import pytest
import torch

from shadowspill_b200.ops import _lib, attention, reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens, Hq, Hkv, dh, seed):
    """Views of one fused projection, as a decoder layer passes them."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    T = sum(lens)
    qkv = (torch.randn(T, (Hq + 2 * Hkv) * dh, generator=g) * 0.8).to(torch.bfloat16).to(DEV)
    q = qkv[:, :Hq * dh].view(T, Hq, dh)
    k = qkv[:, Hq * dh:(Hq + Hkv) * dh].view(T, Hkv, dh)
    v = qkv[:, (Hq + Hkv) * dh:].view(T, Hkv, dh)
    dout = (torch.randn(T, Hq, dh, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    return q, k, v, dout, cu


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


EDGES = [[1], [127, 128, 129], [255, 256, 257], [64, 63, 65, 384, 1], [640]]


@pytest.mark.parametrize("dh", [64, 128, 256])
@pytest.mark.parametrize("lens", EDGES + [[3 + 17 * i for i in range(40)]], ids=lambda x: f"{len(x)}seq{sum(x)}")
@pytest.mark.parametrize("scale", [None, -0.05])
def test_against_the_definition(lens, dh, scale):
    q, k, v, dout, cu = _inputs(lens, 4, 2, dh, seed=sum(lens))
    out, lse = attention.forward(q, k, v, cu, max(lens), scale)
    dq, dk, dv = attention.backward(q, k, v, out, lse, dout, cu, max(lens), scale)
    _lib.check_status()
    out_r, lse_r = R.attention_varlen(q, k, v, cu, scale)
    dq_r, dk_r, dv_r = R.attention_varlen_bwd(q, k, v, out_r, lse_r, dout, cu, scale)
    # bf16 probabilities and results: 2^-9 relative rounding each, a few such roundings per output
    assert _rel(out, out_r) < 1e-2
    assert float((lse - lse_r).abs().max()) < 1e-3
    # the gradients of a one-token sequence are zero up to cancellation in dP - delta
    if max(lens) > 1:
        assert _rel(dq, dq_r) < 2e-2
        assert _rel(dk, dk_r) < 2e-2
    assert _rel(dv, dv_r) < 2e-2


def test_gradients_repeat_bit_for_bit():
    q, k, v, dout, cu = _inputs([300, 700, 129], 8, 2, 128, seed=5)
    out, lse = attention.forward(q, k, v, cu, 700)
    runs = [attention.backward(q, k, v, out, lse, dout, cu, 700) for _ in range(3)]
    for other in runs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(runs[0], other))


@pytest.mark.parametrize("Hq,Hkv", [(8, 2), (6, 1), (4, 4), (16, 1)])
@pytest.mark.parametrize("dh", [64, 128, 256])
@pytest.mark.parametrize("lens", [[200], [130, 700, 70], [4000, 2700]], ids=lambda x: f"sum{sum(x)}")
def test_groups_shared_by_clusters(lens, dh, Hq, Hkv):
    """Group sizes that are and are not divisible by the cluster sizes, few and many key tiles."""
    q, k, v, dout, cu = _inputs(lens, Hq, Hkv, dh, seed=Hq + dh)
    out, lse = attention.forward(q, k, v, cu, max(lens))
    dq, dk, dv = attention.backward(q, k, v, out, lse, dout, cu, max(lens))
    again = attention.backward(q, k, v, out, lse, dout, cu, max(lens))
    _lib.check_status()
    assert all(torch.equal(a, b) for a, b in zip((dq, dk, dv), again))
    out_r, lse_r = R.attention_varlen(q, k, v, cu)
    dq_r, dk_r, dv_r = R.attention_varlen_bwd(q, k, v, out_r, lse_r, dout, cu)
    assert _rel(dq, dq_r) < 2e-2 and _rel(dk, dk_r) < 2e-2 and _rel(dv, dv_r) < 2e-2


@pytest.mark.parametrize("width", [64, 128, 256])
def test_results_do_not_depend_on_other_work_on_the_gpu(width):
    # work of another stream on the same SMs slows some warps of a tile: those that are a step ahead must
    # neither count for the others nor be lapped by the products that wait for them
    from shadowspill_b200.ops import functional as F
    lens = [128, 200, 100, 128, 450, 128, 60, 128, 256, 120] * 6
    T, H, Hk = sum(lens), 32, 8
    g = torch.Generator(device="cuda").manual_seed(width)
    q, k, v, do = (torch.randn(T, h, width, generator=g, device="cuda").to(torch.bfloat16) for h in (H, Hk, Hk, H))
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    alone = F.attention_varlen(q, k, v, cu, max(lens))
    torch.cuda.synchronize()
    grads = F.attention_varlen_bwd(q, k, v, *alone, do, cu, max(lens))
    torch.cuda.synchronize()
    side, noise = torch.cuda.Stream(), torch.randn(148 * 4 * 1024, device="cuda")
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(40):
        with torch.cuda.stream(side):
            for _ in range(6):
                noise.sin_()
        out = F.attention_varlen(q, k, v, cu, max(lens))
        outs.append((*out, *F.attention_varlen_bwd(q, k, v, *alone, do, cu, max(lens))))
    torch.cuda.synchronize()
    _lib.check_status()
    for got in outs:
        for a, b in zip(got, (*alone, *grads)):
            assert torch.equal(a, b)


def _growing_in_one_quarter(dh, quarter):
    """Scores that grow by 2^11.5 with every 64 keys, in one 32-row quarter of each 128-row tile: its warp
    moves its reference maximum at every step and waits for the product before, the others never do."""
    lens = [700, 64, 513, 1000, 257]
    q, k, v, dout, cu = _inputs(lens, 8, 2, dh, seed=dh + quarter)
    q, k = q.contiguous(), k.contiguous()
    at = torch.cat([torch.arange(n) for n in lens]).to(DEV)           # position in its sequence
    q[:, :, 0] = torch.where(at % 128 // 32 == quarter, 16.0, 0.0)[:, None].to(q.dtype)
    k[:, :, 0] = (at // 64 * 4)[:, None].to(k.dtype)
    return q, k, v, dout, cu, max(lens), 0.125


def _beside_other_work(run, repeats=30):
    """Results of ``run()`` while another stream's blocks share the SMs with its warps."""
    torch.cuda.synchronize()
    side, noise = torch.cuda.Stream(), torch.randn(148 * 4 * 1024, device=DEV)
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(repeats):
        with torch.cuda.stream(side):
            for _ in range(6):
                noise.sin_()
        outs.append(run())
    torch.cuda.synchronize()
    _lib.check_status()
    return outs


@pytest.mark.parametrize("quarter", [0, 2])
@pytest.mark.parametrize("dh", [64, 128, 256])
def test_forward_with_one_warp_behind(dh, quarter):
    # a warp that has finished a step must not count for one of the same tile that has not
    q, k, v, _, cu, longest, scale = _growing_in_one_quarter(dh, quarter)
    out, lse = attention.forward(q, k, v, cu, longest, scale)
    _lib.check_status()
    out_r, lse_r = R.attention_varlen(q, k, v, cu, scale)
    assert _rel(out, out_r) < 1e-2                                    # bf16 probabilities and results
    assert float((lse - lse_r).abs().max()) < 1e-3
    for got in _beside_other_work(lambda: attention.forward(q, k, v, cu, longest, scale)):
        assert torch.equal(got[0], out) and torch.equal(got[1], lse)


def _gradients_beside_other_work(dh):
    q, k, v, dout, cu, longest, scale = _growing_in_one_quarter(dh, 1)
    out, lse = attention.forward(q, k, v, cu, longest, scale)
    run = lambda: attention.backward(q, k, v, out, lse, dout, cu, longest, scale)  # noqa: E731
    grads = run()
    _lib.check_status()
    out_r, lse_r = R.attention_varlen(q, k, v, cu, scale)
    for a, b in zip(grads, R.attention_varlen_bwd(q, k, v, out_r, lse_r, dout, cu, scale)):
        assert _rel(a, b) < 2e-2
    for got in _beside_other_work(run):
        assert all(torch.equal(a, b) for a, b in zip(got, grads))


@pytest.mark.parametrize("dh", [64, 128])
def test_backward_with_warps_a_tile_apart(dh):
    # scores and dP of the next key tile are ready before the slowest warp has written dS of this one
    _gradients_beside_other_work(dh)


def test_wide_backward_with_warps_a_tile_apart():
    # dV alone: scores of the next query tile are ready before the slowest warp has written P^T of this one
    _gradients_beside_other_work(256)


def test_more_sequences_than_a_grid_has_rows():
    """66,000 one-token sequences, past the 65,535 of a grid's second dimension, and one of 200 tokens."""
    n, tail, dh = 66000, 200, 64
    g = torch.Generator().manual_seed(3)
    q, k, v, dout = (torch.randn(n + tail, 1, dh, generator=g).to(torch.bfloat16).to(DEV) for _ in range(4))
    cu = torch.tensor([*range(n + 1), n + tail], dtype=torch.int32, device=DEV)
    out, lse = attention.forward(q, k, v, cu, tail)
    dq, dk, dv = attention.backward(q, k, v, out, lse, dout, cu, tail)
    _lib.check_status()
    assert torch.equal(out[:n], v[:n]) and torch.equal(dv[:n], dout[:n])          # one key: probability one
    assert torch.allclose(lse[0, :n], (q[:n].float() * k[:n].float()).sum((1, 2)) / 8, rtol=1e-5, atol=1e-4)
    # dP and delta are the same sum in two orders: what is left of their difference is fp32 rounding
    assert float(dq[:n].abs().max()) < 1e-4 and float(dk[:n].abs().max()) < 1e-4
    one = torch.tensor([0, tail], dtype=torch.int32, device=DEV)
    rest = [t[n:] for t in (q, k, v)]
    out_r, lse_r = R.attention_varlen(*rest, one)
    grads_r = R.attention_varlen_bwd(*rest, out_r, lse_r, dout[n:], one)
    assert _rel(out[n:], out_r) < 1e-2
    for a, b in zip((dq, dk, dv), grads_r):
        assert _rel(a[n:], b) < 2e-2


@pytest.mark.parametrize("dh", [64, 128, 256])
@pytest.mark.parametrize("shift", [2, 4, 6])
def test_saved_output_off_a_sixteen_byte_boundary(dh, shift):
    q, k, v, dout, cu = _inputs([130, 77], 4, 2, dh, seed=dh + shift)
    out, lse = attention.forward(q, k, v, cu, 130)
    moved = torch.empty(out.numel() + 8, dtype=out.dtype, device=DEV)[shift:shift + out.numel()].view(out.shape)
    moved.copy_(out)
    assert moved.data_ptr() % 16 == 2 * shift
    want = attention.backward(q, k, v, out, lse, dout, cu, 130)
    got = attention.backward(q, k, v, moved, lse, dout, cu, 130)
    _lib.check_status()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
