"""AdamW of many tensors in shared launches: the bits of one call per tensor, at the edges of vectors,
blocks, the launch's table and the size that still shares a launch."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"
HYPER = dict(lr=3e-3, beta1=0.9, beta2=0.95, eps=1e-8, weight_decay=0.1, step=3, grad_scale=0.5, seed=11)
EDGES = [1, 7, 8, 9, 2040, 2047, 2048, 2049, 4096, 100003, F.ADAMW_MANY_ELEMENTS - 1, F.ADAMW_MANY_ELEMENTS,
         F.ADAMW_MANY_ELEMENTS + 1]


def _tensors(sizes):
    g = torch.Generator(device=DEV).manual_seed(len(sizes))
    r = lambda n, s: torch.randn(n, generator=g, device=DEV) * s
    out, offset = [], 0
    for i, n in enumerate(sizes):
        grad = r(n, 1e-2) if i % 3 == 1 else r(n, 1e-2).bfloat16()
        out.append((r(n, 0.1).bfloat16(), grad, r(n, 1e-2).bfloat16(), r(n, 1e-2).square().bfloat16(), offset))
        offset += (n + 7) // 8 * 8
    return out


@pytest.mark.parametrize("sizes", [EDGES, [257] * 39, [65] * 40, [513] * 41, [4100] * 83, [0, 5, 0, 24], [0]],
                         ids=["edges", "39", "40", "41", "83", "empty", "none"])
@pytest.mark.parametrize("sr", [(True, True), (False, True), (True, False), (False, False)])
def test_many_tensors_have_the_bits_of_single_calls(sizes, sr):
    flags = dict(stochastic_param=sr[0], stochastic_state=sr[1])
    one, many = _tensors(sizes), _tensors(sizes)
    for p, g, m, v, offset in one:
        F.adamw_(p, g, m, v, offset=offset, **HYPER, **flags)
    F.adamw_many_(many, **HYPER, **flags)
    for a, b in zip(one, many):
        for x, y in zip(a[:4], b[:4]):
            assert torch.equal(x, y)


def test_a_tensor_listed_twice_and_fp32_parameters():
    def lists():
        a = _tensors([300, 40, 9])
        f = tuple(t.float() for t in a[1][:4]) + (0,)
        return [a[0], a[1], a[0], f, a[2], a[0]]
    one, many = lists(), lists()
    for p, g, m, v, offset in one:
        F.adamw_(p, g, m, v, offset=offset, **HYPER)
    F.adamw_many_(many, **HYPER)
    for a, b in zip(one, many):
        assert all(torch.equal(x, y) for x, y in zip(a[:4], b[:4]))


def test_offsets_off_the_vector_are_refused():
    p, g, m, v, _ = _tensors([64])[0]
    with pytest.raises(RuntimeError):
        F.adamw_many_([(p, g, m, v, 4)], **HYPER)
