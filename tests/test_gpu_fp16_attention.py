"""fp32 attention in fp16 pieces (csrc/flash_x2.cu) at the edges of its tiles, and the heads that it leaves to the kernels behind it,
against the row-group kernels (configuration 1) and 64 bits."""
import pytest

pytestmark = pytest.mark.gpu


def inputs(cuda, B, T, NH, hs, seed):
    C = NH * hs
    g = cuda.Generator(device="cuda").manual_seed(seed)
    return cuda.randn(B, T, 3 * C, generator=g, device="cuda"), cuda.randn(B, T, C, generator=g, device="cuda")


def attention(bmb, cuda, cfg, qkv, dout, NH, lse_add=0.0):
    B, T, C = dout.shape
    out, lse, dsum, dqkv = (cuda.full(s, float("nan"), device="cuda") for s in ((B, T, C), (B, NH, T), (B, NH, T), (B, T, 3 * C)))
    bmb.call("bmb_flash_attention_forward_cfg", cfg, out, lse, qkv, B, T, C, NH)
    bmb.call("bmb_flash_attention_backward_cfg", cfg, dqkv, dsum, dout, qkv, out, lse + lse_add, B, T, C, NH)
    cuda.cuda.synchronize()
    return out, lse, dsum, dqkv


def relative(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


# One head of 64-bit errors up to 3e-7 (tests of split attention), so two fp32 implementations are up to 8e-7 apart.
BOUND = 1e-6


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("B,T,NH", [(1, 512, 1), (1, 513, 2), (2, 575, 1), (1, 640, 3), (1, 641, 1), (1, 767, 1), (1, 833, 2), (3, 1025, 1),
                                    (20, 512, 8)])                 # the last: more pairs of tiles than SMs
def test_edges_of_tiles(bmb, cuda, hs, B, T, NH):
    qkv, dout = inputs(cuda, B, T, NH, hs, T + hs)
    for x, y in zip(attention(bmb, cuda, 0, qkv, dout, NH), attention(bmb, cuda, 1, qkv, dout, NH)):
        assert bool(cuda.isfinite(x).all()) and relative(x, y) <= BOUND
    again = attention(bmb, cuda, 0, qkv, dout, NH)
    assert all(cuda.equal(x, y) for x, y in zip(again, attention(bmb, cuda, 0, qkv, dout, NH)))


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("what", ["tiny", "huge", "a row", "inf", "nan", "zero"])
@pytest.mark.parametrize("which", [0, 1, 2, 3])
def test_heads_that_the_pieces_cannot_serve(bmb, cuda, hs, what, which):
    """One of four heads has a block of 64 positions out of range; it and the others come out as they do from the row groups."""
    B, T, NH = 2, 520, 2
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, 7 * hs + which)
    block = (dout if which == 3 else qkv[..., which * C:(which + 1) * C])[1, 128:192, hs:2 * hs]
    if what == "tiny":
        block *= 2.0 ** -60
    elif what == "huge":
        block *= 2.0 ** 40 if which > 1 else 2.0 ** 3
    elif what == "a row":
        block[5] *= 2.0 ** -30
    elif what == "zero":
        block.zero_()
    else:
        block[5, 3] = float(what)
    if what == "huge" and which < 2:
        block *= 2.0 ** 28
        (qkv[..., (1 - which) * C:(2 - which) * C])[1, :, hs:2 * hs] *= 2.0 ** -31
    got, want = attention(bmb, cuda, 0, qkv, dout, NH), attention(bmb, cuda, 1, qkv, dout, NH)
    heads = lambda x: x.reshape(B, T, -1, hs).transpose(1, 2).reshape(B, -1, NH, T, hs) if x.shape[1] == T else x    # noqa: E731
    for x, y in zip(got, want):
        assert cuda.equal(cuda.isfinite(x), cuda.isfinite(y)) and cuda.equal(cuda.isnan(x), cuda.isnan(y))
        for a, b in zip(heads(x).unbind(0), heads(y).unbind(0)):
            fin = cuda.isfinite(b)
            scale = cuda.where(fin, b, cuda.zeros_like(b)).abs().max()
            if scale > 0:
                assert float((cuda.where(fin, a - b, cuda.zeros_like(a)) / scale).norm() / cuda.where(fin, b / scale, cuda.zeros_like(b)).norm()) <= BOUND


@pytest.mark.parametrize("hs", [32, 64, 128])
def test_lse_of_other_scores(bmb, cuda, hs):
    """Probabilities beyond 1 (an lse that is not these scores') are beyond what the pieces are scaled for."""
    qkv, dout = inputs(cuda, 1, 512, 2, hs, hs)
    got, want = attention(bmb, cuda, 0, qkv, dout, 2, -6.0), attention(bmb, cuda, 1, qkv, dout, 2, -6.0)
    assert relative(got[3], want[3]) <= BOUND


def test_captured_calls(bmb, cuda):
    """A caller's capture holds no address of the library's scratch; the captured call gives what an eager one gives."""
    B, T, NH, hs = 1, 512, 2, 64
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, 3)
    eager = attention(bmb, cuda, 0, qkv, dout, NH)
    out, lse = cuda.empty(B, T, C, device="cuda"), cuda.empty(B, NH, T, device="cuda")
    stream = cuda.cuda.Stream()
    graph = cuda.cuda.CUDAGraph()
    with cuda.cuda.stream(stream):
        with cuda.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            bmb.lib().bmb_set_stream(cuda.cuda.current_stream().cuda_stream)
            bmb.call("bmb_flash_attention_forward_cfg", 0, out, lse, qkv, B, T, C, NH)
    bmb.lib().bmb_set_stream(None)
    graph.replay()
    cuda.cuda.synchronize()
    assert relative(out, eager[0]) <= BOUND and relative(lse, eager[1]) <= BOUND


def in_64_bits(cuda, qkv, dout, NH):
    """out, lse, and dq, dk, dv as (B, NH, T, hs)."""
    B, T, C = dout.shape
    hs = C // NH
    heads = lambda x: x.double().reshape(B, T, NH, hs).transpose(1, 2)      # noqa: E731
    (q, k, v), do = (heads(x) for x in qkv.chunk(3, dim=-1)), heads(dout)
    s = (q @ k.transpose(2, 3) / hs ** 0.5).masked_fill(cuda.ones(T, T, dtype=cuda.bool, device="cuda").triu(1), float("-inf"))
    lse = cuda.logsumexp(s, -1)
    p = cuda.exp(s - lse[..., None])
    out = p @ v
    ds = p * (do @ v.transpose(2, 3) - (do * out).sum(-1, keepdim=True)) / hs ** 0.5
    return out, lse, ds @ k, ds.transpose(2, 3) @ q, p.transpose(2, 3) @ do


def by_heads(cuda, got, NH):
    out, lse, _, dqkv = got
    heads = lambda x: x.unflatten(-1, (NH, -1)).transpose(1, 2)      # noqa: E731
    return heads(out), lse, *(heads(x) for x in dqkv.chunk(3, dim=-1))


def no_worse(cuda, bmb, qkv, dout, NH, parts):
    """Errors against 64 bits of parts of the five results are at most twice the row groups' (or within BOUND: theirs are sums of 32 terms
    in a row, so their errors vary by less than that with the order).  parts: (result, index of its head and rows)."""
    want = in_64_bits(cuda, qkv, dout, NH)
    got, groups = (by_heads(cuda, attention(bmb, cuda, cfg, qkv, dout, NH), NH) for cfg in (0, 1))
    for r, at in parts:
        mine, theirs = relative(got[r][at], want[r][at]), relative(groups[r][at], want[r][at])
        assert mine <= max(BOUND, 2 * theirs), (r, at, mine, theirs)


OUT, LSE, DQ, DK, DV = range(5)


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("which,e", [(2, 0), (2, -7), (2, -14), (2, -20), (3, 0), (3, -14)])
def test_a_block_of_zeros(bmb, cuda, hs, which, e):
    """64 positions whose V (or dO) is zero, where the other blocks are small: dS there is - P D, whatever the size of V."""
    B, T, NH = 1, 640, 2
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, hs)
    x = dout if which == 3 else qkv[..., 2 * C:]
    x *= 2.0 ** e
    x[0, 128:192, hs:2 * hs] = 0
    rows, all_ = slice(128, 192), slice(None)
    parts = [(r, (0, h, all_)) for r in (OUT, LSE, DQ, DK, DV) for h in (0, 1)] + [(r, (0, 1, rows)) for r in (OUT, DK, DV)]
    no_worse(cuda, bmb, qkv, dout, NH, parts + ([(DQ, (0, 1, rows))] if which == 2 else []))


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("size", [1e2, 1e3, 3e3, 1e4, 3e4, 1e5])
@pytest.mark.parametrize("sign", [1, -1])
def test_large_scores(bmb, cuda, hs, size, sign):
    """Scores of 10^4 to 10^10, of mixed and (every query a negative multiple of its key and more) of one sign: a row's weight is on one key."""
    B, T, NH = 1, 640, 2
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, hs)
    if sign < 0:
        qkv[..., :C] = -qkv[..., :C].abs()
        qkv[..., C:2 * C] = qkv[..., C:2 * C].abs()
    qkv[..., :2 * C] *= size
    got, want = (by_heads(cuda, attention(bmb, cuda, cfg, qkv, dout, NH), NH) for cfg in (0, 1))
    assert all(bool(cuda.isfinite(x).all()) for x in got)
    # Scores that are rounded at their size decide between keys that lie that close: such rows differ between any two implementations.
    (q, k) = (x.unflatten(-1, (NH, hs)).transpose(1, 2).double() for x in qkv.chunk(3, dim=-1)[:2])
    s = (q @ k.transpose(2, 3) / hs ** 0.5).masked_fill(cuda.ones(T, T, dtype=cuda.bool, device="cuda").triu(1), float("-inf"))
    two = s.topk(2, dim=-1).values
    clear = (two[..., 0] - two[..., 1]) > 20 + 2.0 ** -18 * s.masked_fill(s.isinf(), 0).abs().amax(-1)
    clear[..., 0] = True
    assert clear.double().mean() > 0.5
    assert relative(got[OUT][clear], want[OUT][clear]) <= BOUND and relative(got[LSE], want[LSE]) <= BOUND


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("shift", [-0.5, -1.0, -30.0, -60.0, -84.0, -100.0, -150.0, -200.0, -300.0])
def test_lse_far_below_the_scores(bmb, cuda, hs, shift):
    """Weights of 1.6 to e^90 come out as from the row groups, and what overflows there is not finite here either.  (An exponential's
    argument, up to |shift| + 12 in natural units, is rounded to 24 bits on either side, and so is its product with log2 e.)"""
    qkv, dout = inputs(cuda, 1, 512, 2, hs, hs)
    got, want = (by_heads(cuda, attention(bmb, cuda, cfg, qkv, dout, 2, shift), 2) for cfg in (0, 1))
    for r in (DQ, DK, DV):
        assert cuda.equal(cuda.isfinite(got[r]), cuda.isfinite(want[r])), r
        fin = cuda.isfinite(want[r])
        if bool(fin.any()):
            assert relative(got[r][fin], want[r][fin]) <= BOUND + 4 * 2.0 ** -24 * (abs(shift) + 12), r


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("which,e", [(w, e) for w in range(4) for e in (-16, -28, -40)])
def test_a_small_column(bmb, cuda, hs, which, e):
    """One column of a head's q, k, v or dO is 2^e of the others: out, dv, dk and dq are sums per column."""
    B, T, NH = 1, 640, 2
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, hs)
    x = dout if which == 3 else qkv[..., which * C:(which + 1) * C]
    x[..., hs + 5] *= 2.0 ** e
    col = (0, 1, slice(None), 5)
    parts = {0: [(DK, col)], 1: [(DQ, col)], 2: [(OUT, col)], 3: [(DV, col)]}[which]
    no_worse(cuda, bmb, qkv, dout, NH, parts + [(r, (0, h, slice(None))) for r in range(5) for h in (0, 1)])


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("e", [11, 13, 19])
def test_rows_beside_large_ones(bmb, cuda, hs, e):
    """A row of V or dO 2^e times the others, which the queries before it or the keys behind it do not see, and one 2^-e of the others."""
    B, T, NH, all_ = 1, 640, 2, slice(None)
    C = NH * hs
    for which, at, size, rows in ((2, 150, e, [(DQ, slice(128, 150)), (OUT, slice(128, 150))]), (3, 600, e, [(DK, slice(601, T)), (DV, slice(601, T))]),
                                  (2, 150, -e, [(DK, slice(150, 151))]), (3, 600, -e, [(DQ, slice(600, 601))]),
                                  (3, T - 1, -e, [(DK, slice(T - 1, T)), (DV, slice(T - 1, T))])):
        qkv, dout = inputs(cuda, B, T, NH, hs, hs)
        (dout if which == 3 else qkv[..., 2 * C:])[0, at, hs:2 * hs] *= 2.0 ** size
        no_worse(cuda, bmb, qkv, dout, NH, [(r, (0, 1, x)) for r, x in rows] + [(r, (0, h, all_)) for r in range(5) for h in (0, 1)])


@pytest.mark.parametrize("hs", [32, 64, 128])
def test_rows_of_zeros(bmb, cuda, hs):
    """Keys whose V and queries whose dO is zero, to the left and right of a block's edge, and all that a row of the block sees."""
    B, T, NH, all_ = 1, 640, 2, slice(None)
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, hs)
    qkv[0, :70, 2 * C + hs:2 * C + 2 * hs] = 0
    qkv[0, 300, 2 * C:2 * C + hs] = 0
    dout[0, 600:, hs:2 * hs] = 0
    dout[0, 300, :hs] = 0
    no_worse(cuda, bmb, qkv, dout, NH, [(r, (0, h, all_)) for r in range(5) for h in (0, 1)])
    got = by_heads(cuda, attention(bmb, cuda, 0, qkv, dout, NH), NH)
    assert all(bool(cuda.isfinite(x).all()) for x in got)
    assert not got[OUT][0, 1, :70].any() and not got[DQ][0, 1, :70].any() and not got[DQ][0, 1, 600:].any()
    assert not got[DK][0, 1, 600:].any() and not got[DV][0, 1, 600:].any() and not got[DQ][0, 0, 300].any()


@pytest.mark.parametrize("hs", [32, 64, 128])
@pytest.mark.parametrize("heads", [[0], [299], [127, 128], [0, 31, 32, 255, 256, 299], range(300)])
def test_some_of_many_heads(bmb, cuda, hs, heads):
    """Heads with a row out of range, among more heads than a block of the kernels behind has threads."""
    B, T, NH = 100, 384, 3
    C = NH * hs
    qkv, dout = inputs(cuda, B, T, NH, hs, hs)
    for i in heads:
        qkv[i // NH, 70, 2 * C + i % NH * hs:2 * C + (i % NH + 1) * hs] *= 2.0 ** -30
    got, want = (by_heads(cuda, attention(bmb, cuda, cfg, qkv, dout, NH), NH) for cfg in (0, 1))
    for x, y in zip(got, want):
        x, y = (z.flatten(0, 1).flatten(1).double() for z in (x, y))
        assert bool(((x - y).norm(dim=1) <= BOUND * y.norm(dim=1)).all())


@pytest.mark.parametrize("B,T,NH,hs", [(9, 8192, 8, 128), (11, 8192, 26, 32), (1, 65600, 9, 128)])
def test_images_in_parts(bmb, cuda, B, T, NH, hs):
    """More heads than images of 1 GiB hold (some sequences at a time, or some heads of one): the first and the last, bit for bit as by themselves."""
    qkv, dout = inputs(cuda, B, T, NH, hs, 1)
    out, lse, dsum, dqkv = attention(bmb, cuda, 0, qkv, dout, NH)
    for b, h in ((0, 0), (B - 1, NH - 1)):
        pick = lambda x: x[b:b + 1].unflatten(-1, (-1, NH, hs))[:, :, :, h].flatten(2).contiguous()      # noqa: E731
        alone = attention(bmb, cuda, 0, pick(qkv), pick(dout), 1)
        for x, y in zip((pick(out), lse[b:b + 1, h:h + 1], dsum[b:b + 1, h:h + 1], pick(dqkv)), alone):
            assert cuda.equal(x, y)


def test_calls_on_several_streams(bmb, cuda):
    """Calls on four streams, of several sizes, without a wait between them: what each gives by itself."""
    shapes = [(1, 512, 4, 64), (2, 777, 12, 32), (1, 1024, 8, 128), (4, 1024, 12, 64)]
    data = [inputs(cuda, *shape, i) for i, shape in enumerate(shapes)]
    want = [attention(bmb, cuda, 0, qkv, dout, shape[2]) for shape, (qkv, dout) in zip(shapes, data)]
    streams = [cuda.cuda.Stream() for _ in shapes]
    got = [[cuda.full_like(x, float("nan")) for x in w] for w in want]
    cuda.cuda.synchronize()
    try:
        for _ in range(20):
            for st, (B, T, NH, hs), (qkv, dout), (out, lse, dsum, dqkv) in zip(streams, shapes, data, got):
                bmb.lib().bmb_set_stream(st.cuda_stream)
                bmb.call("bmb_flash_attention_forward_cfg", 0, out, lse, qkv, B, T, NH * hs, NH)
                bmb.call("bmb_flash_attention_backward_cfg", 0, dqkv, dsum, dout, qkv, out, lse, B, T, NH * hs, NH)
    finally:
        bmb.lib().bmb_set_stream(None)
    cuda.cuda.synchronize()
    assert all(cuda.equal(x, y) for g, w in zip(got, want) for x, y in zip(g, w))


def test_calls_of_several_threads(bmb, cuda):
    """Four threads, each with its stream of the one handle cudaStreamPerThread, on blocks of several sizes: what each gives by itself."""
    import threading
    shapes = [(1, 512, 4, 64), (2, 777, 12, 32), (1, 1024, 8, 128), (4, 1024, 12, 64)]
    data = [inputs(cuda, *shape, i) for i, shape in enumerate(shapes)]
    want = [attention(bmb, cuda, 0, qkv, dout, shape[2]) for shape, (qkv, dout) in zip(shapes, data)]
    got = [[cuda.full_like(x, float("nan")) for x in w] for w in want]
    cuda.cuda.synchronize()
    failed = []

    def work(i):
        (B, T, NH, hs), (qkv, dout), (out, lse, dsum, dqkv) = shapes[i], data[i], got[i]
        try:
            bmb.lib().bmb_set_stream(2)                # cudaStreamPerThread
            for _ in range(20):
                bmb.call("bmb_flash_attention_forward_cfg", 0, out, lse, qkv, B, T, NH * hs, NH)
                bmb.call("bmb_flash_attention_backward_cfg", 0, dqkv, dsum, dout, qkv, out, lse, B, T, NH * hs, NH)
        except Exception as e:
            failed.append(e)
        finally:
            bmb.lib().bmb_set_stream(None)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    cuda.cuda.synchronize()
    assert not failed
    assert all(cuda.equal(x, y) for g, w in zip(got, want) for x, y in zip(g, w))
