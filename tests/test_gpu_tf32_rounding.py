"""TF32 products that round their operands where they land in shared memory (csrc/gemm_tc.cu, RND), against the same
products of operands rounded beforehand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NO_SPLIT, A_ROUNDED, B_ROUNDED = 8, 1, 2


def rounded(torch, x):
    """cvt.rna.tf32: half an ulp of 10 mantissa bits added to the magnitude, the rest cut; NaN stays NaN."""
    u = x.view(torch.int32)
    return torch.where(torch.isnan(x), x, ((u + 0x1000) & ~0x1fff).view(torch.float32))


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(128, 64, 32), (132, 68, 36), (256, 256, 256), (1000, 300, 100), (200, 1000, 2000), (3000, 96, 500)])
def test_rounding_on_arrival_equals_the_pass(bmb, cuda, M, N, K, ta, tb):
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    A, B = (cuda.randn(s, generator=g, device="cuda") for s in ((K, M) if ta else (M, K), (N, K) if tb else (K, N)))
    a = A.T if ta else A
    a[3, 1], a[5, 2], a[7, 3] = float("inf"), float("nan"), 3.4e38            # the last rounds to infinity
    a[9, 4] = cuda.tensor(0x7fffffff, dtype=cuda.int32).view(cuda.float32)    # a NaN that an addition would carry out of
    C = [cuda.full((M, N), float("nan"), device="cuda") for _ in range(2)]
    bmb.call("bmb_gemm_ex", bmb.MATH_TF32, NO_SPLIT, ta, tb, M, N, K, 1.0, A, B, 0.0, C[0], None)
    bmb.call("bmb_gemm_ex", bmb.MATH_TF32, NO_SPLIT | A_ROUNDED | B_ROUNDED, ta, tb, M, N, K, 1.0, rounded(cuda, A), rounded(cuda, B), 0.0, C[1], None)
    cuda.cuda.synchronize()
    x, y = (c.cpu().numpy() for c in C)
    assert np.isnan(y[5]).all() and np.isnan(y[9]).all() and np.isfinite(y[11:]).all()
    assert np.array_equal(x, y, equal_nan=True)


def test_rounding_on_arrival_of_batches(bmb, cuda):
    n, T, hs = 5, 192, 64
    g = cuda.Generator(device="cuda").manual_seed(3)
    q, k, p = (cuda.randn(s, generator=g, device="cuda") for s in ((n, T, hs), (n, T, hs), (n, T, T)))
    prev = bmb.lib().bmb_get_math_mode()
    bmb.lib().bmb_set_math_mode(bmb.MATH_TF32)
    out = []
    for f in (lambda x: x, lambda x: rounded(cuda, x)):
        s, o = cuda.empty(n, T, T, device="cuda"), cuda.empty(n, T, hs, device="cuda")
        bmb.call("bmb_batched_gemm", 0, 1, n, T, T, hs, 0.125, f(q), T * hs, f(k), T * hs, 0.0, s, T * T, None)
        bmb.call("bmb_batched_gemm", 0, 0, n, T, hs, T, 1.0, f(p), T * T, f(k), T * hs, 0.0, o, T * hs, None)
        out += [s, o]
    bmb.lib().bmb_set_math_mode(prev)
    cuda.cuda.synchronize()
    assert cuda.equal(out[0], out[2]) and cuda.equal(out[1], out[3])
    want = rounded(cuda, q).double() @ rounded(cuda, k).double().transpose(1, 2) * 0.125
    assert float((out[0].double() - want).norm() / want.norm()) < 2e-6


# One launch (and one that prepares shared tiles) where operands are rounded on arrival, up to two passes more where not.
@pytest.mark.parametrize("M,N,K,flags,beta,launches", [
    (128, 64, 32, NO_SPLIT, 0.0, 1),
    (132, 68, 36, NO_SPLIT, 0.0, 1),
    (1000, 300, 100, NO_SPLIT, 0.0, 1),
    (1024, 1024, 256, 0, 0.0, 1),
    (200, 1000, 2000, 0, 0.0, 2),            # tiles shared along K: their sums start from beta C, written by a launch before
    (768, 768, 4096, 0, 0.0, 2),
    (768, 768, 4096, 0, 0.5, 2),
    (768, 768, 4096, 0, 1.0, 1),
    (6144, 128, 6144, 0, 0.0, 2),
    (200, 1000, 2000, NO_SPLIT, 0.0, 3),     # here the passes cost less
    (2048, 2048, 2048, NO_SPLIT, 0.0, 3),
    (4096, 4096, 4096, NO_SPLIT, 0.0, 3),
])
def test_where_operands_are_rounded_on_arrival(bmb, cuda, M, N, K, flags, beta, launches):
    """The route, by the launches it takes, and the result against the 64-bit product of rounded operands: the tensor core cuts
    its sum off at each of K / 8 instructions, at most 2^-23 of a running sum that is no larger than its end is in the mean."""
    g = cuda.Generator(device="cuda").manual_seed(M + K)
    A, B, C0 = (cuda.randn(s, generator=g, device="cuda") for s in ((M, K), (K, N), (M, N)))
    C = C0.clone()
    before = bmb.lib().bmb_launch_count()
    bmb.call("bmb_gemm_ex", bmb.MATH_TF32, flags, 0, 0, M, N, K, 1.0, A, B, beta, C, None)
    assert bmb.lib().bmb_launch_count() - before == launches
    cuda.cuda.synchronize()
    want = rounded(cuda, A).double() @ rounded(cuda, B).double() + beta * C0.double()
    assert float((C.double() - want).norm() / want.norm()) < K / 8 * 2.0 ** -23
