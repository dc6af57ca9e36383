"""RMSNorm kernels over row widths at the edges of their forms (8-lane rows to 12288 channels), row
counts from one to more than a grid, residual add and accumulation, and heads in place of a projection."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F, reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"
EPS = 1e-5


def _rand(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g) * std).to(torch.bfloat16).to(DEV)


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


# one bf16 rounding of the result is 2^-9 relative at most; fp32 sums of up to 12288 terms add ~1e-6
TOL = 4e-3


@pytest.mark.parametrize("D", [8, 64, 72, 128, 136, 256, 264, 512, 520, 1024, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("T", [1, 37, 1300])
@pytest.mark.parametrize("zc", [False, True])
def test_rows(D, T, zc):
    g = torch.Generator().manual_seed(D * 7 + T)
    x, w, gy, delta = _rand(g, T, D), _rand(g, D), _rand(g, T, D), _rand(g, T, D)
    x1, x2 = x.clone(), x.clone()
    y, rstd = F.rmsnorm_fwd(x1, w, EPS, zc)
    y_r, rstd_r = R.rmsnorm_fwd(x2, w, EPS, zc)
    assert torch.equal(x1, x) and _rel(y, y_r) < TOL and _rel(rstd, rstd_r) < 1e-5
    yd, _ = F.rmsnorm_fwd(x1, w, EPS, zc, delta=delta)
    yd_r, _ = R.rmsnorm_fwd(x2, w, EPS, zc, delta=delta)
    assert torch.equal(x1, x2) and _rel(yd, yd_r) < TOL
    dw = torch.full((D,), 2.0, device=DEV)
    dx = F.rmsnorm_bwd(x, w, gy, rstd_r, dw, zc)
    dx_r, dw_r = R.rmsnorm_bwd(x, w, gy, rstd_r, zc)
    assert _rel(dx, dx_r) < TOL and _rel(dw - 2.0, dw_r) < 1e-4
    into = gy.clone()
    F.rmsnorm_bwd(x, w, gy, rstd_r, None, zc, dx=into, accumulate=True)
    assert _rel(into, dx_r + gy.float()) < TOL


@pytest.mark.parametrize("D,T", [(8200, 300), (12288, 500)])
def test_widest_backward(D, T):
    g = torch.Generator().manual_seed(D)
    x, w, gy = _rand(g, T, D), _rand(g, D), _rand(g, T, D)
    rstd = torch.rsqrt(x.float().square().mean(-1) + EPS)
    dw, dx = torch.zeros(D, device=DEV), gy.clone()
    F.rmsnorm_bwd(x, w, gy, rstd, dw, False, dx=dx, accumulate=True)
    dx_r, dw_r = R.rmsnorm_bwd(x, w, gy, rstd, False)
    assert _rel(dx, dx_r + gy.float()) < TOL and _rel(dw, dw_r) < 1e-4


@pytest.mark.parametrize("dh", [32, 64, 128, 256])
@pytest.mark.parametrize("T,heads,rest", [(1, 1, 0), (129, 6, 3), (700, 16, 16)])
def test_heads_in_place(dh, T, heads, rest):
    g = torch.Generator().manual_seed(dh + T)
    buf, w, d = _rand(g, T, (heads + rest) * dh), _rand(g, dh), _rand(g, T, (heads + rest) * dh)
    n = heads * dh
    before, tail, dtail = buf[:, :n].clone(), buf[:, n:].clone(), d[:, n:].clone()
    raw = torch.empty_like(buf)
    rstd = F.head_norm_(buf[:, :n], w, heads, EPS, raw=raw[:, :n])
    y_r, rstd_r = R.rmsnorm_fwd(before.reshape(T * heads, dh), w, EPS)
    assert torch.equal(raw[:, :n], before) and torch.equal(buf[:, n:], tail)
    assert _rel(buf[:, :n], y_r.view(T, n)) < TOL and _rel(rstd, rstd_r) < 1e-5
    gy, dw = d[:, :n].clone(), torch.zeros(dh, device=DEV)
    F.head_norm_bwd_(raw[:, :n], w, d[:, :n], rstd, dw, heads)
    dx_r, dw_r = R.rmsnorm_bwd(before.reshape(T * heads, dh), w, gy.reshape(T * heads, dh), rstd)
    assert _rel(d[:, :n], dx_r.view(T, n)) < TOL and _rel(dw, dw_r) < 1e-4
    assert torch.equal(d[:, n:], dtail)
    _lib.check_status()


@pytest.mark.parametrize("D", [64, 128, 256, 512, 1024, 2048, 4096, 8192])
def test_fused_residual_add_gives_the_same_bits(D):
    """One frontend folds the residual add into the norm and another adds first: same results."""
    g = torch.Generator().manual_seed(D)
    x, w, delta = _rand(g, 300, D), _rand(g, D), _rand(g, 300, D)
    added = x + delta
    y, rstd = F.rmsnorm_fwd(added.clone(), w, EPS)
    folded = x.clone()
    y2, rstd2 = F.rmsnorm_fwd(folded, w, EPS, delta=delta)
    assert torch.equal(folded, added) and torch.equal(y, y2) and torch.equal(rstd, rstd2)


@pytest.mark.parametrize("D", [64, 256, 512, 2048, 4096, 8200])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_weight_gradient_off_a_sixteen_byte_boundary(D, shift):
    """A view into a flat fp32 buffer may start at any element."""
    g = torch.Generator().manual_seed(D + shift)
    x, w, gy = _rand(g, 150, D), _rand(g, D), _rand(g, 150, D)
    rstd = torch.rsqrt(x.float().square().mean(-1) + EPS)
    flat = torch.full((D + 8,), 3.0, device=DEV)
    dw = flat[shift:shift + D]
    assert dw.data_ptr() % 16 == 4 * shift
    F.rmsnorm_bwd(x, w, gy, rstd, dw)
    dx_r, dw_r = R.rmsnorm_bwd(x, w, gy, rstd)
    assert _rel(dw - 3.0, dw_r) < 1e-4
    assert bool((flat[:shift] == 3.0).all()) and bool((flat[shift + D:] == 3.0).all())
    if D <= 512:
        dw.fill_(0.0)
        d = gy.repeat(1, 2).contiguous()
        F.head_norm_bwd_(x.repeat(1, 2).contiguous(), w, d, rstd.repeat_interleave(2), dw, 2)
        assert _rel(dw, 2.0 * dw_r.float()) < 1e-4 and _rel(d[:, :D], dx_r) < TOL
    _lib.check_status()
