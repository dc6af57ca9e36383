"""The GEMMs with SwiGLU or a residual in their epilogue against the separate kernels, whose bits they have to have."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(*shape, std=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * std).bfloat16()


# rows and widths around the tiles of the three kernels: one wave of 128 x 128, CTA pairs, ragged edges
SHAPES = [(1, 64, 128), (127, 256, 64), (300, 520, 192), (768, 1024, 256), (1999, 6144, 2048), (2049, 1032, 520)]


@pytest.mark.parametrize("T,Ff,D", SHAPES)
def test_fused_swiglu_has_the_bits_of_the_separate_kernels(T, Ff, D):
    x, w13, w2, dy = _rand(T, D, seed=1), _rand(2 * Ff, D, std=0.1, seed=2), _rand(D, Ff, std=0.1, seed=3), _rand(T, D, seed=4)
    gu = F.linear_fwd(x, w13)
    h = F.swiglu_fwd(gu)
    got_gu, got_h = F.swiglu_linear(x, w13)
    none, alone = F.swiglu_linear(x, w13, keep_gu=False)
    assert none is None and torch.equal(got_gu, gu) and torch.equal(got_h, h) and torch.equal(alone, h)
    wide_gu, wide_h = (torch.zeros(T, n + 8, dtype=gu.dtype, device=DEV) for n in (2 * Ff, Ff))
    F.swiglu_linear(x, w13, gu=wide_gu[:, :2 * Ff], out=wide_h[:, :Ff])            # pitches wider than the rows
    assert torch.equal(wide_gu[:, :2 * Ff], gu) and torch.equal(wide_h[:, :Ff], h)
    assert float(wide_gu[:, 2 * Ff:].abs().max()) == 0.0 == float(wide_h[:, Ff:].abs().max())
    dgu = F.swiglu_bwd(gu, F.linear_dgrad(dy, w2))
    assert torch.equal(F.swiglu_linear_dgrad(dy, w2, gu), dgu)
    _lib.check_status()


@pytest.mark.parametrize("T,Ff,D", SHAPES)
def test_a_residual_is_added_with_the_bits_of_a_copy(T, Ff, D):
    h, w2, x = _rand(T, Ff, seed=5), _rand(D, Ff, std=0.1, seed=6), _rand(T, D, seed=7)
    want = F.linear_fwd(h, w2, out=x.clone(), accumulate=True)
    kept = x.clone()
    assert torch.equal(F.linear_residual(h, w2, x), want) and torch.equal(x, kept)
    out = torch.empty_like(x)
    assert F.linear_residual(h, w2, x, out=out) is out and torch.equal(out, want)
    assert torch.equal(F.linear_residual(h, w2, x, out=x), want)


def test_operands_the_fused_forms_do_not_take_go_through_the_separate_ones():
    x, w13 = _rand(130, 64, seed=1), _rand(40, 64, seed=2)                        # 20 columns of each: not pieces of eight
    with pytest.raises(ValueError):
        F.swiglu_linear(x[:, ::2], w13[:, ::2])                                   # refused as before: inner stride
    gu, h = F.swiglu_linear(x, w13[:32])
    assert torch.equal(h, F.swiglu_fwd(F.linear_fwd(x, w13[:32]))) and torch.equal(gu, F.linear_fwd(x, w13[:32]))


def test_the_expert_form_has_the_bits_of_the_separate_kernels():
    from shadowspill_b200.ops import moe
    E, T, D, Ff, k = 8, 300, 256, 192, 2
    x, bank = _rand(T, D, seed=1), _rand(E, 2 * Ff, D, std=0.1, seed=2)
    ids, wts, counts = moe.route(torch.randn(T, E, device=DEV), k, True)
    lay = moe.Layout(ids, counts)
    xs = lay.gather(x)
    used = int(lay.used)
    gu = moe.grouped_linear(xs, bank, lay)
    got_gu, got_h = moe.grouped_swiglu(xs, bank, lay)
    assert torch.equal(got_gu[:used], gu[:used]) and torch.equal(got_h[:used], lay.swiglu(gu)[:used])


def test_a_residual_with_nothing_to_add_is_the_residual():
    x, w, res = _rand(300, 8)[:, :0], _rand(256, 8)[:, :0], _rand(300, 256, seed=1)
    out = torch.full_like(res, float("nan"))
    assert F.linear_residual(x, w, res, out=out) is out and torch.equal(out, res)
    assert torch.equal(F.linear_residual(x, w, res), res)
