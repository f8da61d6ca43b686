"""fp32 SIMT products in tiles of 64 and 32 (csrc/gemm_simt_small.cu): the same sequential chains as the 128-wide
kernels, bit for bit the CPU oracle's, at edges of tiles and slices, aligned and not."""
import numpy as np
import pytest
from helpers import _np, uniform

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("batch,M,N,K", [
    (1, 1, 1, 1), (1, 31, 33, 32), (1, 32, 64, 4), (1, 100, 70, 33), (1, 65, 130, 128),      # tiles of 32
    (12, 256, 256, 96), (3, 500, 400, 100), (2, 513, 385, 129), (1, 960, 64, 97),            # and of 64, K from 96
    (5, 64, 68, 31), (2, 36, 1000, 64), (1, 3, 2000, 130)])
def test_small_tiles_follow_the_sequential_chain(bmb, orc, cuda, ta, tb, batch, M, N, K):
    A, B = uniform(batch * M * K, 1), uniform(batch * K * N, 2)
    want = np.zeros(batch * M * N, np.float32)
    orc.orc_batched_gemm(ta, tb, batch, M, N, K, 1.0, _np(A), M * K, _np(B), K * N, 0.0, _np(want), M * N)
    for offset in (0, 1):                      # 16-byte aligned operands, and operands one float off
        dA, dB = (cuda.zeros(x.size + 4, device="cuda") for x in (A, B))
        dA[offset:offset + A.size], dB[offset:offset + B.size] = cuda.from_numpy(A).cuda(), cuda.from_numpy(B).cuda()
        dC = cuda.full((batch * M * N,), float("nan"), device="cuda")
        prev = bmb.lib().bmb_get_math_mode()
        bmb.lib().bmb_set_math_mode(bmb.MATH_FP32)
        bmb.call("bmb_batched_gemm", ta, tb, batch, M, N, K, 1.0, dA[offset:], M * K, dB[offset:], K * N, 0.0, dC, M * N, None)
        bmb.lib().bmb_set_math_mode(prev)
        cuda.cuda.synchronize()
        assert np.array_equal(dC.cpu().numpy(), want), offset


@pytest.mark.parametrize("M,N,K", [(256, 1152, 384), (70, 132, 33), (33, 64, 97), (1, 4, 1), (257, 700, 130)])
def test_bias_and_gelu_ride_with_the_product(bmb, cuda, M, N, K):
    """X W^T + bias and its GELU from one launch have the bits of the three passes (tiles of 64 x 32 and of 32)."""
    A, W, bias = (cuda.from_numpy(uniform(n, i)).cuda() for i, n in enumerate((M * K, N * K, N)))
    want, want_gelu, got, gelu = (cuda.full((M * N,), float("nan"), device="cuda") for _ in range(4))
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 1, M, N, K, 1.0, A, W, 0.0, want, None)
    bmb.call("bmb_bias_forward", want, bias, M, N)
    bmb.call("bmb_gelu_forward", want_gelu, want, M * N)
    bmb.call("bmb_gemm_bias_gelu", bmb.MATH_FP32, 0, M, N, K, A, W, bias, got, gelu, None)
    cuda.cuda.synchronize()
    assert cuda.equal(got, want) and cuda.equal(gelu, want_gelu)


@pytest.mark.parametrize("M,N,K", [(70, 132, 33), (33, 64, 97), (1, 4, 1), (130, 68, 40)])
@pytest.mark.parametrize("rounded,in_place", [(True, False), (False, True), (True, True)])
def test_rounded_and_in_place(bmb, cuda, M, N, K, rounded, in_place):
    """The passes behind a product round what they store where the activation is asked for rounded, the sum with the bias included, and
    the activation may take the product's place."""
    A, W, bias = (cuda.from_numpy(uniform(n, i)).cuda() for i, n in enumerate((M * K, N * K, N)))
    want, want_gelu, got = (cuda.full((M * N,), float("nan"), device="cuda") for _ in range(3))
    gelu = got if in_place else cuda.full((M * N,), float("nan"), device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 1, M, N, K, 1.0, A, W, 0.0, want, None)
    bmb.call("bmb_bias_forward", want, bias, M, N)
    if rounded:
        bmb.call("bmb_round_tf32", want, want, M * N, None)
    bmb.call("bmb_gelu_forward", want_gelu, want, M * N)
    if rounded:
        bmb.call("bmb_round_tf32", want_gelu, want_gelu, M * N, None)
    bmb.call("bmb_gemm_bias_gelu", bmb.MATH_FP32, bmb.GEMM_AUX_ROUNDED if rounded else 0, M, N, K, A, W, bias, got, gelu, None)
    cuda.cuda.synchronize()
    assert cuda.equal(gelu, want_gelu) and (in_place or cuda.equal(got, want))
