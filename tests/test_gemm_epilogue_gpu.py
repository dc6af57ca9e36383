"""GEMM outputs at the edges of the epilogue's 32 x 16 blocks, written and accumulated, bf16 and fp32,
into a wider buffer whose other columns must not change; both GEMM kernels."""
import pytest
import torch

from shadowspill_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 31, 128, 161, 255, 257, 400])
@pytest.mark.parametrize("N", [8, 24, 128, 136, 264, 520])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_edges(M, N, dtype):
    g = torch.Generator().manual_seed(M * 1000 + N)
    K = 72
    a = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    wide = torch.randn(M, N + 16, generator=g).to(dtype).cuda()
    before = wide.clone()
    out = wide[:, 8:8 + N]
    ref = a.double() @ b.double().t()
    # one rounding to the output type (2^-9 for bf16) on top of fp32 sums of 72 products
    tol = 4e-3 if dtype == torch.bfloat16 else 1e-5
    scale = float(ref.abs().max())
    F.gemm(a, b, out=out, alpha=0.5)
    assert float((out.double() - 0.5 * ref).abs().max()) <= tol * scale
    first = out.clone()
    F.gemm(a, b, out=out, accumulate=True)
    assert float((out.double() - (first.double() + ref)).abs().max()) <= 2 * tol * scale
    assert torch.equal(wide[:, :8], before[:, :8]) and torch.equal(wide[:, 8 + N:], before[:, 8 + N:])
    if M >= 256 and N > 128:                          # the pair kernel, which one SM pair's grid selects
        ldc = wide.stride(0)
        wide.copy_(before)
        _lib.check(_lib.lib().ss_gemm2_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), M, N, K, K, K, ldc, 0, 0,
                                            int(dtype == torch.float32), 1, 2.0, 2, _lib.status_ptr(a),
                                            _lib.stream_ptr()), "ss_gemm2_bf16")
        want = before[:, 8:8 + N].double() + 2.0 * ref
        assert float((out.double() - want).abs().max()) <= 2 * tol * scale
        assert torch.equal(wide[:, :8], before[:, :8]) and torch.equal(wide[:, 8 + N:], before[:, 8 + N:])
    _lib.check_status()


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(257, 136, 72), (1000, 520, 328), (513, 264, 40), (256, 512, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("accumulate", [False, True])
def test_pair_kernel_layouts(a_mn, b_mn, M, N, K, dtype, accumulate):
    """The pair kernel with both operand orders at sizes with remainders: on two SMs, as an output whose
    128 x 128 tiles fit one wave of the whole GPU goes to the other kernel."""
    g = torch.Generator().manual_seed(M + N + K)
    pad = lambda n: -(-n // 8) * 8                                         # noqa: E731  row strides: 16-byte pieces
    a_buf = torch.randn(*((K, pad(M)) if a_mn else (M, pad(K))), generator=g).to(torch.bfloat16).cuda()
    b_buf = torch.randn(*((K, pad(N)) if b_mn else (N, pad(K))), generator=g).to(torch.bfloat16).cuda()
    a = a_buf[:, :M].t() if a_mn else a_buf[:, :K]
    b = b_buf[:, :N].t() if b_mn else b_buf[:, :K]
    wide = torch.randn(M, N + 16, generator=g).to(dtype).cuda()
    before, out = wide.clone(), wide[:, 8:8 + N]
    _lib.check(_lib.lib().ss_gemm2_bf16(a_buf.data_ptr(), b_buf.data_ptr(), out.data_ptr(), M, N, K, a_buf.stride(0),
                                        b_buf.stride(0), wide.stride(0), int(a_mn), int(b_mn), int(dtype == torch.float32),
                                        int(accumulate), 0.5, 2, _lib.status_ptr(a_buf), _lib.stream_ptr()), "ss_gemm2_bf16")
    _lib.check_status()
    want = 0.5 * (a.double() @ b.double().t()) + (before[:, 8:8 + N].double() if accumulate else 0.0)
    # one rounding to the output type (2^-9 for bf16) on top of fp32 sums of up to 328 products
    tol = 4e-3 if dtype == torch.bfloat16 else 1e-5
    assert float((out.double() - want).abs().max()) <= tol * float(want.abs().max())
    assert torch.equal(wide[:, :8], before[:, :8]) and torch.equal(wide[:, 8 + N:], before[:, 8 + N:])
