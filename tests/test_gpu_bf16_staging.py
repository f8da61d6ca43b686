"""BF16 products: the converted copies of the operands (csrc/gemm_tc.cu) by 128-bit words and by the general routes."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(128, 128, 40), (132, 196, 72), (1000, 1004, 1000), (513, 1000, 777), (300, 2001, 68), (644, 130, 100)])
def test_bf16_product_of_rounded_operands(bmb, cuda, M, N, K, ta, tb):
    """Against the 64-bit product of the operands rounded to bf16: what is left is the fp32 accumulation, cut off once per
    16 K at 2^-24 of the sum, below 2^-23 * K / 16 in all."""
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: cuda.rand(s, generator=g, device="cuda") * 2 - 1      # noqa: E731
    A, B = rnd(*((K, M) if ta else (M, K))), rnd(*((N, K) if tb else (K, N)))
    C = cuda.full((M, N), float("nan"), device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_BF16, 0, ta, tb, M, N, K, 1.0, A, B, 0.0, C, None)
    cuda.cuda.synchronize()
    want = (A.T if ta else A).bfloat16().double() @ (B.T if tb else B).bfloat16().double()
    assert float((C.double() - want).norm() / want.norm()) < max(4, K / 16) * 2.0 ** -23
