"""The delta rule's state walks at one chunk, two, an odd number and a ragged end, with one, two, an
odd number and several V heads per key head, forward and backward against the token recurrence."""
import pytest
import torch

from shadowspill_b200.ops import _lib, delta_rule

pytestmark = pytest.mark.gpu


def _recurrence(q, k, v, beta, g, cu):
    rep = v.shape[1] // q.shape[1]
    q, k = (t.repeat_interleave(rep, 1) for t in (q, k))
    out = []
    starts = set(cu)
    for t in range(v.shape[0]):
        if t in starts:
            S = torch.zeros(v.shape[1], 128, 128, dtype=v.dtype, device=v.device)
        S = S * g[t].exp()[:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hk,hkv->hv", k[t], S))
        S = S + k[t][:, :, None] * u[:, None, :]
        out.append(torch.einsum("hk,hkv->hv", q[t], S) * 128 ** -0.5)
    return torch.stack(out)


@pytest.mark.parametrize("T,cu", [(1, [0]), (64, [0]), (65, [0, 30]), (128, [0, 64]), (323, [0, 5, 200])])
@pytest.mark.parametrize("Hk,H", [(1, 1), (2, 4), (1, 3), (1, 4)])
def test_against_the_recurrence(T, cu, Hk, H):
    gen = torch.Generator(device="cuda").manual_seed(T * 10 + H)
    rn = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(rn(T, Hk, 128), dim=-1).bfloat16() for _ in range(2))
    v, dout = rn(T, H, 128).bfloat16(), (0.1 * rn(T, H, 128)).bfloat16()
    beta, g = torch.sigmoid(rn(T, H)), -0.2 * torch.nn.functional.softplus(rn(T, H))
    ends = torch.tensor([*cu, T], dtype=torch.int32, device="cuda")
    leaves = [t.detach().requires_grad_(True) for t in (q, k, v, beta, g)]
    out = delta_rule.gated_delta_rule(*leaves, ends)
    grads = torch.autograd.grad(out, leaves, dout)
    _lib.check_status()
    exact = [t.double().requires_grad_(True) for t in (q, k, v, beta, g)]
    ref = _recurrence(*exact, cu)
    wanted = torch.autograd.grad(ref, exact, dout.double())
    # bf16 operands of chained products: a handful of 2^-9 roundings
    for got, want in zip((out, *grads), (ref, *wanted)):
        assert float((got.double() - want).norm()) <= 1.5e-2 * float(want.norm()) + 1e-6
