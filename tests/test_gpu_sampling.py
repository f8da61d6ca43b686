"""Sampling in fp32: the next token's distribution from one sequence's rows, and text drawn one position at a time with
the keys and values of earlier positions in place, against the model in 64 bits (plain torch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Model64:
    def __init__(self, torch, t):
        c = t.cfg
        w = torch.empty(t.num_params)
        t.get_params(w)
        w *= 3                                     # tokens as different as a trained model tells them apart
        t.set_params(w)
        self.torch, self.c, C, L, at = torch, c, c.n_embd, c.n_layer, 0
        self.p = []
        for shape in [(c.padded_vocab, C), (c.max_seq_len, C), (L, C), (L, C), (L, 3 * C, C), (L, 3 * C), (L, C, C), (L, C), (L, C), (L, C),
                      (L, 4 * C, C), (L, 4 * C), (L, C, 4 * C), (L, C), (C,), (C,)]:
            n = int(np.prod(shape))
            self.p.append(w[at:at + n].reshape(shape).cuda().double())
            at += n
        assert at == t.num_params

    def probs(self, tokens):
        torch, F, c = self.torch, self.torch.nn.functional, self.c
        wte, wpe, l1w, l1b, qw, qb, aw, ab, l2w, l2b, fw, fb, pw, pb, lw, lb = self.p
        n, C, NH = len(tokens), c.n_embd, c.n_head
        x = wte[torch.as_tensor(tokens, device="cuda").long()] + wpe[:n]
        mask = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
        for i in range(c.n_layer):
            q, k, v = (F.layer_norm(x, (C,), l1w[i], l1b[i]) @ qw[i].T + qb[i]).reshape(n, 3, NH, C // NH).permute(1, 2, 0, 3)
            s = (q @ k.transpose(1, 2) / (C // NH) ** 0.5).masked_fill(mask, float("-inf"))
            x = x + (torch.softmax(s, -1) @ v).transpose(0, 1).reshape(n, C) @ aw[i].T + ab[i]
            h = F.gelu(F.layer_norm(x, (C,), l2w[i], l2b[i]) @ fw[i].T + fb[i], approximate="tanh")
            x = x + h @ pw[i].T + pb[i]
        logits = F.layer_norm(x[-1], (C,), lw, lb) @ wte.T
        return torch.softmax(logits[:c.vocab_size], -1).cpu().numpy()


CONFIGS = [  # heads, head size, B, T, vocabulary, flash
    (3, 32, 4, 48, 65, 1),
    (2, 64, 1, 70, 300, 1),
    (2, 128, 3, 33, 65, 1),
    (3, 64, 2, 40, 65, 0),
]


@pytest.mark.parametrize("heads,hs,B,T,V,flash", CONFIGS)
def test_sampling_against_64_bits(bmb, cuda, heads, hs, B, T, V, flash):
    Vp = -(-V // 128) * 128
    t = bmb.Trainer(seed=7, max_seq_len=T, vocab_size=V, padded_vocab=Vp, n_layer=3, n_head=heads, n_embd=heads * hs, B=B, T=T,
                    use_flash=flash, math=bmb.MATH_FP32, fused=0)
    m = Model64(cuda, t)
    # Any position of any sequence. A pass over the whole batch with the same chains is up to 2.4e-5 off here (the model
    # amplifies: gains and weights are three times their usual size); 1e-4 is four times that.
    rng = np.random.default_rng(1)
    tokens = rng.integers(0, V, (B, T)).astype(np.int32)
    for b, pos in [(0, 0), (B - 1, 1), (B - 1, T - 1), (B // 2, T // 2)]:
        got = cuda.empty(Vp)
        bmb.call("bmb_trainer_next_token_probs", t.h, tokens, b * T + pos, got)
        want = m.probs(tokens[b, :pos + 1])
        assert np.abs(got.numpy()[:V] / want - 1).max() < 1e-4 and not got.numpy()[V:].any()
    # a text longer than the context: positions one by one, then the sliding window, by the same coins
    steps, seed, temperature = T + 9, 11, 0.8
    text = t.generate(0, steps, seed, temperature)
    coins = np.random.RandomState(seed).randint(0, 2 ** 32, size=steps, dtype=np.uint32).astype(np.float32) / np.float32(2 ** 32)
    ctx = [0]
    for s in range(steps):
        p = m.probs(ctx[-T:]) ** (1 / temperature)
        cdf = np.cumsum(p / p.sum())
        tok = min(int(np.searchsorted(cdf, coins[s], side="right")), V - 1)
        if tok != text[s]:                         # only a coin within rounding of a step of the distribution may differ
            assert np.abs(cdf - coins[s]).min() < 1e-5, (s, tok, text[s])
            tok = text[s]
        ctx.append(tok)
    # a step of training after it is unchanged by what sampling left in the buffers
    t.upload(tokens, tokens)
    t.step(0.0, 1)
    loss = t.loss()
    t.step(0.0, 2)
    assert abs(t.loss() - loss) < 1e-6
    t.close()


@pytest.mark.parametrize("heads,hs,T,layers", [
    (2, 32, 300, 2),        # more than 256 positions: the running maximum is carried from one 32 groups of keys to the next
    (1, 128, 400, 1),       # more than 320 at 128 columns (and 640 at 64): the values no longer fit in shared memory
    (2, 64, 700, 1),
    (9, 32, 70, 2),         # 1152 inputs: the ring of weight slices comes round
])
def test_long_texts_position_by_position(bmb, cuda, heads, hs, T, layers):
    """Texts that fill the context, drawn one position at a time. The distributions of the window path, which follows the same
    order of sums, choose the same tokens by the same coins; they themselves are within 1e-4 of the model in 64 bits."""
    V, Vp, B = 65, 128, 2
    t = bmb.Trainer(seed=5, max_seq_len=T, vocab_size=V, padded_vocab=Vp, n_layer=layers, n_head=heads, n_embd=heads * hs, B=B, T=T,
                    use_flash=1, math=bmb.MATH_FP32, fused=0)
    m = Model64(cuda, t)
    seed = 3
    text = t.generate(0, T - 1, seed, 1.0)
    coins = np.random.RandomState(seed).randint(0, 2 ** 32, size=T - 1, dtype=np.uint32).astype(np.float32) / np.float32(2 ** 32)
    tokens = np.zeros((B, T), np.int32)
    tokens[0, 1:] = text
    got = cuda.empty(Vp)
    for s in list(range(0, T - 1, 7)) + list(range(T - 12, T - 1)):
        bmb.call("bmb_trainer_next_token_probs", t.h, tokens, s, got)
        p = got.numpy()[:V].astype(np.float64)
        cdf = np.cumsum(p / p.sum())
        tok = min(int(np.searchsorted(cdf, coins[s], side="right")), V - 1)
        assert tok == text[s] or np.abs(cdf - coins[s]).min() < 1e-6, (s, tok, text[s])     # (sums of 65 fp32 numbers)
        if s % 49 == 0 or s == T - 2:
            assert np.abs(p / m.probs(tokens[0, :s + 1]) - 1).max() < 1e-4, s
    t.close()


@pytest.mark.parametrize("heads,hs,T,layers", [
    (25, 32, 24, 2),        # 800 channels: 225 tiles of 32 outputs a layer, up to two a block, slices of 128 and of 32 inputs
    (8, 128, 20, 2),        # the widest: 288 tiles, up to three a block, 4096 inputs
    (1, 32, 20, 3),         # the narrowest: 9 tiles, one slice of 32 inputs
])
def test_several_tiles_a_block(bmb, cuda, heads, hs, T, layers):
    test_long_texts_position_by_position(bmb, cuda, heads, hs, T, layers)
