"""Products that the tensor-core modes leave to the fp32 kernels (fewer than 128 rows or 64 columns): the sequential chain,
without scratch, so that captured steps of several trainers on one device may run beside one another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("math", ["MATH_TF32", "MATH_BF16"])
def test_small_products_of_the_tensor_core_modes_follow_the_chain(bmb, cuda, math):
    M, N, K = 100, 4096, 256
    g = cuda.Generator(device="cuda").manual_seed(1)
    A, B = (cuda.randn(s, generator=g, device="cuda") for s in ((M, K), (K, N)))
    C, want = cuda.empty(M, N, device="cuda"), cuda.empty(M, N, device="cuda")
    bmb.call("bmb_gemm_ex", getattr(bmb, math), 0, 0, 0, M, N, K, 1.0, A, B, 0.0, C, None)
    bmb.call("bmb_sgemm_simt", M, N, K, 1.0, A, B, 0.0, want)
    cuda.cuda.synchronize()
    assert cuda.equal(C, want)


@pytest.mark.parametrize("math,fused", [("MATH_TF32", 0), ("MATH_TF32", 1), ("MATH_BF16", 0), ("MATH_FP32", 0)])
def test_trainers_of_one_device_do_not_disturb_each_other(bmb, cuda, math, fused):
    """Two trainers of C = 64 (weight gradients of 64 rows), their captured steps in flight together: the gradients are
    those of each alone.  Learning rate 0, so every step has the same ones; atomic sums of shared tiles may come in
    another order, which leaves 1e-5 of the norm as the bar (BF16: a rounding of an operand that such an order turns over,
    2^-9 of it, so 1e-2)."""
    B, T, V = 4, 128, 65
    cfg = dict(max_seq_len=T, vocab_size=V, padded_vocab=128, n_layer=2, n_head=1, n_embd=64, B=B, T=T, use_flash=1,
               math=getattr(bmb, math), fused=fused)
    rng = np.random.default_rng(3)
    trainers, alone, work = [bmb.Trainer(seed=s, **cfg) for s in (1, 2)], [], []
    for t in trainers:
        tok = [cuda.from_numpy(rng.integers(0, V, (B, T)).astype(np.int32)).pin_memory() for _ in range(2)]
        work.append(tok)
        for step in (1, 2, 3):
            t.upload(*tok)
            t.step(0.0, step)
        g = cuda.empty(t.num_params)
        t.get_grads(g)
        alone.append(g.double())
    for step in range(4, 40):
        for t, tok in zip(trainers, work):
            t.upload(*tok)
            t.step(0.0, step)
    for t, want in zip(trainers, alone):
        g = cuda.empty(t.num_params)
        t.get_grads(g)
        assert float(want.norm()) > 0 and float((g.double() - want).norm() / want.norm()) < (1e-2 if math == "MATH_BF16" else 1e-5)
        t.close()
