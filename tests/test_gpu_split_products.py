"""fp32 products and attention on the tensor cores, every fp32 operand in pieces (csrc/gemm_x3.cu), at the sizes where
the split can go wrong: edges of tiles and slices, K shared among CTAs, infinities and NaN, a stream being captured."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GEMMS = [  # M, N, K, ta, tb, beta
    (512, 512, 192, 0, 1, 0.0),      # the smallest that the rule takes
    (515, 511, 193, 0, 0, 0.5),      # nothing aligned, one K past a slice
    (515, 511, 1025, 1, 1, 0.0),
    (1000, 514, 2047, 1, 0, 1.0),    # K shared among CTAs, even N off 16 bytes
    (33, 8191, 999, 0, 1, 0.0),      # one ragged row tile
    (4100, 68, 1000, 1, 0, 0.0),     # one narrow column tile
    (4100, 4101, 130, 0, 0, -1.0),   # short K, nothing aligned
    (2048, 1536, 512, 0, 1, 0.0),
]


@pytest.mark.parametrize("M,N,K,ta,tb,beta", GEMMS)
def test_split_product_against_64_bits(bmb, cuda, M, N, K, ta, tb, beta):
    """The pieces leave out 2^-26 of each product, a slice's sum in tensor memory is cut off twice at full size (2^-24
    each) and every 32 K one rounding is added: below 4 * 2^-24 = 2.4e-7 of the result in the 2-norm up to K = 2048, and
    below the SIMT kernel's own error."""
    g = cuda.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: cuda.rand(s, generator=g, device="cuda") * 2 - 1      # noqa: E731
    A, B, C0 = rnd(*((K, M) if ta else (M, K))), rnd(*((N, K) if tb else (K, N))), rnd(M, N)
    a, b = (A.T if ta else A), (B.T if tb else B)
    want = 0.75 * (a.double() @ b.double()) + beta * C0.double()
    C = C0.clone() if beta else cuda.full((M, N), float("nan"), device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, ta, tb, M, N, K, 0.75, A, B, beta, C, None)
    simt = C0.clone()
    bmb.call("bmb_sgemm_simt", M, N, K, 0.75, a.contiguous(), b.contiguous(), beta, simt)
    cuda.cuda.synchronize()
    err = lambda x: float((x.double() - want).norm() / want.norm())        # noqa: E731
    assert not cuda.equal(C, simt)                                         # it was the split product that ran
    assert err(C) < 2.4e-7 and err(C) < err(simt), (err(C), err(simt))
    again = C0.clone()
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, ta, tb, M, N, K, 0.75, A, B, beta, again, None)
    cuda.cuda.synchronize()
    assert cuda.equal(C, again)


@pytest.mark.parametrize("M,N,K", [(515, 511, 1025), (2048, 1536, 512)])       # parts of K added by a pass, and whole tiles
def test_split_product_of_infinities_and_nan(bmb, cuda, M, N, K):
    """Where an element is not finite in the sequential chain it is the same here, and operands at the end of the range
    (where the first piece would round to infinity) still give finite results."""
    g = cuda.Generator(device="cuda").manual_seed(5)
    A, B = (cuda.rand(s, generator=g, device="cuda") * 2 - 1 for s in ((M, K), (K, N)))
    A[3, 5], A[7, 0], A[9, 1], A[9, 2], A[M - 1, K - 1] = float("inf"), float("-inf"), float("inf"), float("-inf"), float("nan")
    B[5, 11], B[K - 1, N - 1], B[5, 12] = float("-inf"), float("inf"), 0.0
    A[20], B[:, 20] = 0.0, 0.0
    A[20, 4], B[4, 21] = 3.4028234e38, 0.5
    C, simt = cuda.empty(M, N, device="cuda"), cuda.empty(M, N, device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, C, None)
    bmb.call("bmb_sgemm_simt", M, N, K, 1.0, A, B, 0.0, simt)
    cuda.cuda.synchronize()
    c, s = C.cpu().numpy(), simt.cpu().numpy()
    assert np.isnan(s).any() and np.isinf(s).any()
    assert np.array_equal(np.isnan(c), np.isnan(s)) and np.array_equal(np.isinf(c), np.isinf(s))
    assert np.array_equal(c[np.isinf(s)], s[np.isinf(s)])
    assert abs(c[20, 21] / 1.7014117e38 - 1) < 1e-6


@pytest.mark.parametrize("M,N,K,ta,tb,beta", [
    (515, 511, 1025, 0, 1, 0.5),     # the parts of K added by a pass, nothing aligned
    (512, 516, 2048, 1, 0, 1.0),     # and in words
    (2048, 1536, 512, 0, 0, 0.5),    # whole tiles, with an old value that must be read once
    (1300, 4100, 200, 1, 1, -1.0),   # ragged tiles
    (4100, 68, 1000, 0, 0, 0.0),     # narrow ones
])
def test_infinities_all_over_follow_the_chain(bmb, cuda, M, N, K, ta, tb, beta):
    """Every third row of A holds an infinity and every 50th column of B a NaN: what is not finite in the sequential chain is
    the same here, and the rest is within what a split product differs from the chain (both are below 1e-6 in the 2-norm)."""
    g = cuda.Generator(device="cuda").manual_seed(M + N)
    A, B, C0 = (cuda.rand(s, generator=g, device="cuda") + 0.5 for s in ((M, K), (K, N), (M, N)))
    A[::3, K // 2], B[K - 1, ::50] = float("inf"), float("nan")
    B[K // 2, 7] = -1.0
    C, want = C0.clone(), C0.clone()
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, ta, tb, M, N, K, 0.5, A.T.contiguous() if ta else A, B.T.contiguous() if tb else B, beta, C, None)
    bmb.call("bmb_sgemm_simt", M, N, K, 0.5, A, B, beta, want)
    cuda.cuda.synchronize()
    assert bool(cuda.isinf(want[0, 1:50]).all()) and float(want[0, 7]) == float("-inf") and bool(cuda.isnan(want[:, 0]).all())
    assert cuda.equal(cuda.isnan(C), cuda.isnan(want)) and cuda.equal(cuda.isinf(C), cuda.isinf(want))
    ok, inf = cuda.isfinite(want), cuda.isinf(want)
    assert cuda.equal(C[inf], want[inf]) and bool(ok.any())
    assert float((C[ok] - want[ok]).norm() / want[ok].norm()) < 2e-6


@pytest.mark.parametrize("M,N,K", [(512, 512, 192), (515, 1030, 193), (512, 516, 2048)])       # whole tiles, ragged ones, parts of K
@pytest.mark.parametrize("a,b", [(-104, 104), (-108, 108), (-112, 112), (120, -120), (-126, 126), (-62, -62), (-64, -64), (-70, -62)])
def test_small_operands_keep_their_bits(bmb, cuda, M, N, K, a, b):
    """Operands scaled by 2^a and 2^b: pieces end at 2^-133, and sums of the tensor core at 2^-149.  The error against 64 bits is
    no larger than the sequential chain's."""
    g = cuda.Generator(device="cuda").manual_seed(K)
    A, B = ((cuda.rand(s, generator=g, device="cuda") * 2 - 1) * 2.0 ** e for s, e in (((M, K), a), ((K, N), b)))
    want = A.double() @ B.double()
    C, simt = cuda.empty(M, N, device="cuda"), cuda.empty(M, N, device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, C, None)
    bmb.call("bmb_sgemm_simt", M, N, K, 1.0, A, B, 0.0, simt)
    cuda.cuda.synchronize()
    scale = float(want.norm())
    err = lambda x: float((x.double() - want).norm()) / scale               # noqa: E731
    assert 0 < err(simt) and err(C) <= err(simt), (err(C), err(simt))


def test_one_small_row_and_column(bmb, cuda):
    """A row and a column of small numbers among ordinary ones, old values read once: the rest stays a split product."""
    M, N, K = 512, 768, 256
    g = cuda.Generator(device="cuda").manual_seed(1)
    A, B, C0 = (cuda.rand(s, generator=g, device="cuda") * 2 - 1 for s in ((M, K), (K, N), (M, N)))
    A[70] *= 2.0 ** -118
    B[:, 500] *= 2.0 ** -118
    want = A.double() @ B.double() + 0.5 * C0.double()
    C, simt, plain = C0.clone(), C0.clone(), cuda.empty(M, N, device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.5, C, None)
    bmb.call("bmb_sgemm_simt", M, N, K, 1.0, A, B, 0.5, simt)
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, plain, None)
    cuda.cuda.synchronize()
    assert float((C.double() - want).norm() / want.norm()) < 2.4e-7
    assert cuda.equal(C[64:96], simt[64:96]) and cuda.equal(C[:, 500], simt[:, 500]) and not cuda.equal(C[200:], simt[200:])
    exact = A[70].double() @ B.double()
    assert float((plain[70].double() - exact).norm() / exact.norm()) < 1e-6


def test_a_long_product_of_infinities_ends(bmb, cuda):
    """A tile's sums are all computed again at K = 65536: no wait of the kernel's may depend on that."""
    M, N, K = 1536, 3072, 65536
    A, B, C = cuda.ones(M, K, device="cuda"), cuda.ones(K, N, device="cuda"), cuda.zeros(M, N, device="cuda")
    B[0] = float("inf")
    for _ in range(2):
        bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, C, None)
    cuda.cuda.synchronize()
    bmb.call("bmb_kernel_status", None)
    assert bool((C == float("inf")).all())
    bmb.call("bmb_gemm_ex", bmb.MATH_TF32, 0, 0, 0, 256, 256, 256, 1.0, A, A, 0.0, C, None)      # (fails if a wait had run out)
    cuda.cuda.synchronize()


def test_split_product_stays_out_of_a_capture(bmb, cuda):
    """A caller's captured products take no scratch (its address would be kept, and branches of the graph would share it)."""
    n = 1024
    A, B = cuda.rand(n, n, device="cuda"), cuda.rand(n, n, device="cuda")
    C, want = cuda.zeros(n, n, device="cuda"), cuda.zeros(n, n, device="cuda")
    bmb.call("bmb_sgemm_simt", n, n, n, 1.0, A, B, 0.0, want)
    cuda.cuda.synchronize()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.graph(graph):
        bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, n, n, n, 1.0, A, B, 0.0, C, cuda.cuda.current_stream().cuda_stream)
    graph.replay()
    cuda.cuda.synchronize()
    assert cuda.equal(C, want)


def attention(bmb, cuda, cfg, qkv, dout, B, T, C, NH):
    nan = lambda *s: cuda.full(s, float("nan"), device="cuda")             # noqa: E731
    out, lse, dsum, dqkv = nan(B, T, C), nan(B, NH, T), nan(B, NH, T), nan(B, T, 3 * C)
    bmb.call("bmb_flash_attention_forward_cfg", cfg, out, lse, qkv, B, T, C, NH)
    bmb.call("bmb_flash_attention_backward_cfg", cfg, dqkv, dsum, dout, qkv, out, lse, B, T, C, NH)
    cuda.cuda.synchronize()
    return out, lse, dqkv


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("T", [1, 17, 31, 32, 33, 64, 65, 127, 129, 200, 257])     # blocks of 64 / 128 rows, 32 of the other side
def test_split_attention_against_64_bits(bmb, cuda, hs, T):
    """Every output row is a sum of products exact to 2^-23 in chains cut off twice: below 2^-21 = 4.8e-7 in the 2-norm,
    dq and dk (differences of such sums) below 2^-20."""
    B, NH = 2, 3
    C = NH * hs
    g = cuda.Generator(device="cuda").manual_seed(T * 1000 + hs)
    qkv, dout = cuda.randn(B, T, 3 * C, generator=g, device="cuda"), cuda.randn(B, T, C, generator=g, device="cuda")
    got = attention(bmb, cuda, 0, qkv, dout, B, T, C, NH)
    heads = lambda x: x.double().reshape(B, T, NH, hs).transpose(1, 2)      # noqa: E731
    rows = lambda x: x.transpose(1, 2).reshape(B, T, C)                     # noqa: E731
    (q, k, v), do = (heads(x) for x in qkv.chunk(3, dim=-1)), heads(dout)
    s = (q @ k.transpose(2, 3) / hs ** 0.5).masked_fill(cuda.ones(T, T, dtype=cuda.bool, device="cuda").triu(1), float("-inf"))
    lse = cuda.logsumexp(s, -1)
    p = cuda.exp(s - lse[..., None])
    o = p @ v
    ds = p * (do @ v.transpose(2, 3) - (do * o).sum(-1, keepdim=True)) / hs ** 0.5
    want = [rows(o), lse, rows(ds @ k), rows(ds.transpose(2, 3) @ q), rows(p.transpose(2, 3) @ do)]
    for x, w, bar in zip([got[0], got[1], *got[2].chunk(3, dim=-1)], want, [4.8e-7, 4.8e-7, 9.6e-7, 9.6e-7, 4.8e-7]):
        # a single key: dq and dk are zero but for the rounding of dP - D, so their scale is that of dout
        scale = do.norm() if T == 1 else w.norm()
        assert bool(cuda.isfinite(x).all()) and float((x.double() - w).norm() / scale) < bar


@pytest.mark.parametrize("hs", [32, 64, 128])
def test_split_attention_of_infinities_and_nan(bmb, cuda, hs):
    """Infinite keys (a caller's own mask: probability zero), infinite values, NaN: finite where the row-group kernels
    (config 1) are finite, and equal there."""
    B, T, NH = 1, 200, 2
    C = NH * hs
    g = cuda.Generator(device="cuda").manual_seed(hs)
    qkv, dout = cuda.randn(B, T, 3 * C, generator=g, device="cuda"), cuda.randn(B, T, C, generator=g, device="cuda")
    qkv[0, :, 0] = qkv[0, :, 0].abs() + 1.0
    qkv[0, 70, C] = float("-inf")                 # head 0, key 70: every score -inf
    qkv[0, 150, 2 * C + hs] = float("inf")        # head 1, value 150
    qkv[0, 190, hs + 1] = float("nan")            # head 1, query 190
    new, old = (attention(bmb, cuda, cfg, qkv, dout, B, T, C, NH) for cfg in (0, 1))
    assert bool(cuda.isfinite(old[0][0, :, :hs]).all()) and not bool(cuda.isfinite(old[0]).all())
    for x, y in zip(new[:2], old[:2]):
        assert cuda.equal(cuda.isfinite(x), cuda.isfinite(y)) and cuda.equal(cuda.isnan(x), cuda.isnan(y))
        ok = cuda.isfinite(y)
        assert float((x[ok] - y[ok]).abs().max()) < 1e-5
    # the backward on the same forward results
    res = []
    for cfg in (0, 1):
        dqkv, dsum = cuda.zeros(B, T, 3 * C, device="cuda"), cuda.zeros(B, NH, T, device="cuda")
        bmb.call("bmb_flash_attention_backward_cfg", cfg, dqkv, dsum, dout, qkv, old[0], old[1], B, T, C, NH)
        cuda.cuda.synchronize()
        res.append(dqkv)
    ok = cuda.isfinite(res[1])
    assert cuda.equal(cuda.isfinite(res[0]), ok) and float((res[0][ok] - res[1][ok]).abs().max()) < 2e-5


@pytest.mark.parametrize("per_thread", [False, True])
def test_split_products_of_threads_and_streams_take_turns(bmb, cuda, per_thread):
    """Four threads, a stream each, products of different sizes (the scratch grows under way): each result is what the
    product gives alone.  Also on cudaStreamPerThread: one handle, a stream of its own in each thread."""
    handle = lambda s: 2 if per_thread else s.cuda_stream                  # noqa: E731
    import threading
    shapes = [(1024, 1024, 512), (2048, 1024, 768), (600, 3000, 1000), (1536, 2048, 1024)]
    work, errors = [], []
    for i, (M, N, K) in enumerate(shapes):
        g = cuda.Generator(device="cuda").manual_seed(i)
        A, B = (cuda.rand(s, generator=g, device="cuda") for s in ((M, K), (K, N)))
        alone = cuda.empty(M, N, device="cuda")
        bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, alone, None)
        work.append((M, N, K, A, B, alone, [cuda.empty(M, N, device="cuda") for _ in range(12)], cuda.cuda.Stream()))
    cuda.cuda.synchronize()

    def run(w):
        M, N, K, A, B, _, outs, stream = w
        try:
            for C in outs:
                bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, N, K, 1.0, A, B, 0.0, C, handle(stream))
        except Exception as e:                     # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(w,)) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    cuda.cuda.synchronize()
    assert not errors, errors
    for w in work:
        assert all(cuda.equal(C, w[5]) for C in w[6])


@pytest.mark.parametrize("N,offset", [(514, 0), (516, 1)])
def test_a_bias_that_is_refused_is_refused_at_any_size(bmb, cuda, N, offset):
    """Columns that are no multiple of 4, or a bias off 16 bytes, beside a small product and a split one."""
    g = cuda.zeros(2 ** 20, device="cuda")
    for M, K in [(8, 8), (1024, 512)]:
        with pytest.raises(Exception):
            bmb.call("bmb_gemm_bias_gelu", bmb.MATH_FP32, 0, M, N, K, g, g, g[offset:], cuda.empty(M * N, device="cuda"), cuda.empty(M * N, device="cuda"), None)
    cuda.cuda.synchronize()


def test_growing_the_scratch_leaves_a_capture_alone(bmb, cuda):
    """A product whose images need a larger block than any before, on one stream, while another stream is being captured in
    the global mode: the capture goes on, and both results are right."""
    n = 256
    small, large = cuda.rand(n, n, device="cuda"), [cuda.rand(s, device="cuda") for s in ((3000, 9000), (9000, 3001))]
    C, D, E = cuda.empty(n, n, device="cuda"), cuda.empty(3000, 3001, device="cuda"), cuda.empty(3000, 3001, device="cuda")
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, 600, 600, 600, 1.0, large[0], large[1], 0.0, D, None)      # (a first, small one)
    bmb.call("bmb_sgemm_simt", 3000, 3001, 9000, 1.0, large[0], large[1], 0.0, E)
    side, graph = cuda.cuda.Stream(), cuda.cuda.CUDAGraph()
    cuda.cuda.synchronize()
    with cuda.cuda.graph(graph, capture_error_mode="global"):
        bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, n, n, n, 1.0, small, small, 0.0, C, cuda.cuda.current_stream().cuda_stream)
        bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, 3000, 3001, 9000, 1.0, large[0], large[1], 0.0, D, side.cuda_stream)
    graph.replay()
    cuda.cuda.synchronize()
    assert float((D - E).norm() / E.norm()) < 4e-6 and not cuda.equal(D, E)
    want = cuda.empty_like(C)
    bmb.call("bmb_sgemm_simt", n, n, n, 1.0, small, small, 0.0, want)
    cuda.cuda.synchronize()
    assert cuda.equal(C, want)


def test_large_scratch_is_given_back(bmb, cuda):
    """1.6 GB of images are free again behind the product that took them, and so is a trainer's block behind the trainer."""
    M, K = 2048, 65536
    A, B, C = cuda.rand(M, K, device="cuda"), cuda.rand(K, M, device="cuda"), cuda.empty(M, M, device="cuda")
    free = lambda: (cuda.cuda.synchronize(), cuda.cuda.mem_get_info()[0])[1]      # noqa: E731
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, 512, 512, 512, 1.0, A, B, 0.0, C, None)
    before = free()
    bmb.call("bmb_gemm_ex", bmb.MATH_FP32, 0, 0, 0, M, M, K, 1.0, A, B, 0.0, C, None)
    assert free() > before - (64 << 20)
    want = A[5].double() @ B.double()
    assert float((C[5].double() - want).norm() / want.norm()) < 1e-6
    del A, B, C
    cuda.cuda.empty_cache()
    cfg = dict(max_seq_len=512, vocab_size=20000, padded_vocab=20096, n_layer=1, n_head=4, n_embd=256, B=8, T=512, use_flash=1, math=bmb.MATH_FP32, fused=0)
    tok = np.zeros((8, 512), np.int32)
    before = free()
    for _ in range(2):
        t = bmb.Trainer(seed=1, **cfg)
        for step in (1, 2, 3):
            t.upload(tok, tok)
            t.step(0.0, step)
        t.sync()
        t.close()
        assert free() > before - (8 << 20)
