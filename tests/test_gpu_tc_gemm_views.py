"""The contraction on transposed operands (tc_gemm.cu) against a PyTorch FP32
reference on the same BF16 inputs.

Sizes on the edges: the 64-wide blocks of an MN-major operand (M, N = 32, 64,
65, 128, 136), K not a multiple of 8 where both operands are transposed, K
within and beyond the shallow ring of four stages of 64, a remainder in the last
stage, the 6144 terms up to which views are read in place.  Tolerance: products of BF16 are exact in FP32, so
only the summation order differs: 1e-5 of sum |A||B|, as in test_gpu_tc_gemm.
"""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = [(128, 64, 64), (64, 32, 72), (136, 32, 1000), (32, 32, 1024), (32, 40, 6144), (32, 40, 6152), (200, 136, 4104),
         (64, 2056, 1024), (8, 8, 8)]


@pytest.mark.parametrize("M,N,K", CASES)
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_views_match_reference(lib, M, N, K, ta, tb):
    import surrogate
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 5 * K)
    if ta and tb:
        K += 3  # rows of a transposed operand need no padding
    A = torch.randn(K, M, device="cuda", generator=g).to(torch.bfloat16).t() if ta else \
        torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(K, N, device="cuda", generator=g).to(torch.bfloat16).t() if tb else \
        torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    D = surrogate.gemm_bf16(A, B)
    surrogate.check_kernel_flags()
    ref = (A.double() @ B.double().T).float()
    scale = (A.float().abs() @ B.float().abs().T).max().item()
    assert D.shape == (M, N) and (D - ref).abs().max().item() <= 1e-5 * scale
    again = surrogate.gemm_bf16(A, B)
    assert torch.equal(D, again)
