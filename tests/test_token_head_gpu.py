"""The output head over its scored rows, against the same head in fp32."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F, reference as R, token_head

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(*shape, std=1.0, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return (torch.randn(*shape, generator=g, device=DEV) * std).bfloat16()


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


def _head(rows, h, W, targets, weights, block, dW, accumulate):
    loss = torch.zeros(1, device=DEV)
    hc = rows.take(h)
    dh = torch.empty_like(hc)
    for r0 in range(0, h.shape[0], block):
        r1 = min(h.shape[0], r0 + block)
        logits = rows.logits(hc, W, r0, r1)
        rows.cross_entropy_(logits, targets, weights, loss, r0, r1)
        rows.wgrad(logits, hc, dW, accumulate, r0, r1)
        rows.dgrad(logits, W, dh, r0, r1)
        accumulate = True
    return loss, rows.put(dh)


@pytest.mark.parametrize("T,block", [(700, 256), (2048, 2048), (1025, 500), (3, 2048)])
@pytest.mark.parametrize("mask", ["half", "none", "all", "one", "first block only"])
@pytest.mark.parametrize("accumulate", [False, True])
def test_scored_rows_give_the_head_of_all_rows(T, block, mask, accumulate, monkeypatch):
    V, D = 1000 * 8, 512
    h, W = _rand(T, D, seed=T), _rand(V, D, std=0.05, seed=1)
    g = torch.Generator(device=DEV).manual_seed(7)
    targets = torch.randint(0, V, (T,), generator=g, device=DEV)
    weights = torch.rand(T, generator=g, device=DEV) + 0.1
    keep = {"half": torch.rand(T, generator=g, device=DEV) < 0.5, "none": torch.ones(T, dtype=torch.bool, device=DEV),
            "all": torch.zeros(T, dtype=torch.bool, device=DEV), "one": torch.arange(T, device=DEV) == T - 1,
            "first block only": torch.arange(T, device=DEV) < 65}[mask]
    targets = torch.where(keep, targets, torch.where(torch.arange(T, device=DEV) % 3 == 0, targets, -1))
    weights = torch.where(keep, weights, 0.0)          # masked by the weight, by the target, or by both
    dW = _rand(V, D, std=0.01, seed=2)
    start = dW.clone() if accumulate else torch.zeros_like(dW)
    monkeypatch.setattr(token_head, "MIN_WORK", 0.0)
    rows = token_head.scored(h, W, targets, weights, dW)
    assert isinstance(rows, token_head.ScoredRows)
    loss, dh = _head(rows, h, W, targets, weights, block, dW, accumulate)
    _lib.check_status()
    logits = h.float() @ W.float().t()
    want, _ = R.cross_entropy_(logits, targets, weights)
    assert abs(float(loss) - float(want)) <= 3e-3 * abs(float(want))          # bf16 logits
    ref_dh, ref_dW = logits @ W.float(), logits.t() @ h.float() + start.float()
    assert float(dh[~keep].abs().sum()) == 0.0
    if mask == "all":
        assert float(loss) == 0.0 and torch.equal(dW, start)
        return
    assert _rel(dh, ref_dh) < 1e-2 and _rel(dW, ref_dW) < 1e-2                # bf16 gradients of the logits and results


def test_a_masked_row_of_a_logits_block_is_cleared():
    logits, targets = _rand(5, 4104), torch.tensor([3, -1, 4104, 7, 0], device=DEV)
    weights = torch.tensor([1.0, 1.0, 1.0, 0.0, 2.0], device=DEV)
    want = logits.clone()
    loss, total = torch.zeros(1, device=DEV), R.cross_entropy_(want, targets, weights)[0]
    F.cross_entropy_(logits, targets, weights, loss)
    assert float(logits[1:4].abs().max()) == 0.0
    assert _rel(logits, want) < 1e-2 and abs(float(loss) - float(total)) < 2e-3 * abs(float(total))


@pytest.mark.parametrize("r0,used,R", [(1000, 1010, 300), (500, 505, 100), (500, 512, 500), (100, 192, 64), (64, 70, 80), (500, 400, 70),
                                       (500, 500, 70)])
def test_rows_behind_the_scored_ones_are_cleared_as_deep_as_the_products_read(r0, used, R):
    """The products contract whole steps of 64 rows counted from the block, wherever the block starts in the list; what
    the block's memory held there must not reach them."""
    V, T = 4104, 2048
    slot = object.__new__(token_head.ScoredRows)
    slot.T, slot.V = T, V
    slot.rows = torch.arange(T, dtype=torch.int32, device=DEV)
    slot.count = torch.tensor([used], dtype=torch.int32, device=DEV)
    scored = max(0, min(R, used - r0))
    logits = torch.full((R, V), float("nan"), dtype=torch.bfloat16, device=DEV)
    logits[:scored] = _rand(scored, V)
    targets, weights = torch.zeros(T, dtype=torch.int64, device=DEV), torch.ones(T, device=DEV)
    slot.cross_entropy_(logits, targets, weights, torch.zeros(1, device=DEV), r0, r0 + R)
    depth = min(R, -(-scored // 64) * 64)
    assert not torch.isnan(logits[:depth]).any() and float(logits[scored:depth].abs().sum()) == 0.0
    assert torch.isnan(logits[depth:]).all()                               # nothing past them is touched


@pytest.mark.parametrize("R,D,used", [(700, 512, 130), (1000, 2048, 1000), (1100, 2176, 700), (2048, 2048, 1), (2049, 2056, 1031), (2048, 2048, 0)])
def test_gradients_of_the_scored_rows_have_the_bits_of_all_rows(R, D, used):
    """Outputs of one wave of 128 x 128 tiles and larger ones, which CTA pairs take: the same sums in either."""
    V = 1032
    slot = object.__new__(token_head.ScoredRows)
    slot.T, slot.V = R, V
    slot.count = torch.tensor([300 + used], dtype=torch.int32, device=DEV)
    dlogits, W = _rand(R, V, seed=1), _rand(V, D, seed=2)
    dh = torch.empty(R, D, dtype=torch.bfloat16, device=DEV)
    whole = dh.new_zeros(300 + R, D)
    dlogits[used:] = float("nan")
    slot.dgrad(dlogits, W, whole, 300, 300 + R)
    F.linear_dgrad(dlogits[:max(used, 1)], W, out=dh[:max(used, 1)])
    assert torch.equal(whole[300:300 + used], dh[:used]) and float(whole[:300].abs().sum()) == 0.0
    _lib.check_status()
