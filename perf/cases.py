"""The work this library is timed on, through its public entry points.

A case is a dict of plain values.  Five kinds of work, each from its smallest to its largest use:

  gemm      the registry kernels and gemm(): one product, fp32 / TF32 / BF16, any transposes and sizes
  bgemm     batched_gemm(): the two products of attention over separate heads, scores Q K^T and P V
  flash     fused causal attention, forward and backward, fp32 / TF32, head sizes 32, 64 and 128
  train     a stretch of training through bmb_trainer_*: a few optimiser steps on fresh batches, every loss read,
            and the parameters read back at the end, as for a checkpoint or an evaluation elsewhere
  generate  sampling from a model: a text drawn token by token, and the model's distribution over the next token

prepare() makes what a user's program holds before the call (inputs, outputs to be filled, a trainer); run() is one
pass; work() the bytes and operations a pass cannot do without; tolerance() what two correct implementations of the
same precision may differ by.
"""
import importlib
import math

import numpy as np
import torch

bmb = importlib.import_module("bare-metal-bard_b200")

MATH = {"fp32": bmb.MATH_FP32, "tf32": bmb.MATH_TF32, "bf16": bmb.MATH_BF16}
REGISTRY = {"fp32": "bmb_sgemm_simt", "tf32": "bmb_sgemm_tf32", "bf16": "bmb_sgemm_bf16"}     # C = A B + beta C


# ---- the cases --------------------------------------------------------------------------------------------------

def gemm(math_, M, N, K, ta=0, tb=0, beta=0.0):
    return {"kind": "gemm", "math": math_, "M": M, "N": N, "K": K, "ta": ta, "tb": tb, "beta": beta}


def bgemm(math_, batch, T, hs):
    return {"kind": "bgemm", "math": math_, "batch": batch, "T": T, "hs": hs}


def flash(math_, B, T, NH, hs):
    return {"kind": "flash", "math": math_, "B": B, "T": T, "NH": NH, "hs": hs}


def train(math_, layers, heads, hs, B, T, vocab, steps):
    return {"kind": "train", "math": math_, "layers": layers, "heads": heads, "hs": hs, "B": B, "T": T, "vocab": vocab,
            "steps": steps}


def generate(layers, heads, hs, B, T, vocab, tokens):
    return {"kind": "generate", "math": "fp32", "layers": layers, "heads": heads, "hs": hs, "B": B, "T": T, "vocab": vocab,
            "tokens": tokens}


def listed():
    return [
        # The smallest call: a ragged gemm() with a transposed operand added into its result, as a gradient is.
        # Its launch and its latency are its time.
        dict(gemm("fp32", 100, 70, 33, ta=1, beta=0.5), name="gemm_fp32_ragged_100x70x33"),
        # The single fp32 product of the benchmark configurations (registry entry 1).
        dict(gemm("fp32", 1024, 1024, 1024), name="sgemm_fp32_1024"),
        # A middle point of the registry's size sweep on tensor cores (entry 2), fp32 inputs as the sweep has them.
        dict(gemm("tf32", 4096, 4096, 4096), name="sgemm_tf32_4096"),
        # The sweep's next size in BF16 arithmetic (entry 3), the largest single call listed.
        dict(gemm("bf16", 6144, 6144, 6144), name="sgemm_bf16_6144"),
        # Attention over separate heads at 8 sequences x 12 heads of 1024 tokens: scores, then weights times values.
        dict(bgemm("tf32", 96, 1024, 64), name="bgemm_attention_tf32_96x1024"),
        # Fused attention of the benchmark configuration, forward and backward.
        dict(flash("tf32", 8, 1024, 12, 64), name="flash_tf32_8x1024_h12x64"),
        # Wide heads and a long sequence, forward and backward.
        dict(flash("tf32", 4, 2048, 8, 128), name="flash_tf32_4x2048_h8x128"),
        # The default arithmetic at a length that fills no tile.
        dict(flash("fp32", 2, 777, 12, 32), name="flash_fp32_2x777_h12x32"),
        # Training of the 124M-parameter configuration, the headline benchmark, on tensor cores ...
        dict(train("tf32", 12, 12, 64, 8, 1024, 50304, 8), name="train_124m_tf32"),
        # ... and in the default fp32 arithmetic.
        dict(train("fp32", 12, 12, 64, 8, 1024, 50304, 2), name="train_124m_fp32"),
        # Training at the driver program's default sizes: a character model on one text file.
        dict(train("fp32", 6, 6, 64, 16, 256, 65, 10), name="train_char_fp32"),
        # Sampling a text longer than the context from the same model, as the driver does every few hundred steps.
        dict(generate(6, 6, 64, 16, 256, 65, 300), name="generate_char_fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Log-uniform; a third of the sizes are multiples of 64, a third of 4, a third whatever they are."""
    n = _log_int(rng, lo, hi)
    step = rng.choice((64, 4, 1))
    return max(lo, n // step * step)


def draw(rng):
    kind = rng.choice(("gemm", "gemm", "bgemm", "flash", "flash", "train", "generate"))
    if kind == "gemm":
        return gemm(rng.choice(("fp32", "tf32", "bf16")), _size(rng, 32, 6144), _size(rng, 32, 6144), _size(rng, 32, 6144),
                    rng.randint(0, 1), rng.randint(0, 1), rng.choice((0.0, 0.0, 0.5, 1.0)))
    if kind == "bgemm":
        T = _size(rng, 64, 1024)
        hs = rng.choice((32, 64, 128))
        return bgemm(rng.choice(("fp32", "tf32")), _log_int(rng, 2, 128), T, hs)
    if kind == "flash":
        hs = rng.choice((32, 64, 128))
        T = _size(rng, 64, 2048)
        heads = rng.randint(2, 16)
        B = _log_int(rng, 1, max(2, min(16, 2 ** 17 // (T * heads))))
        return flash(rng.choice(("fp32", "tf32")), B, T, heads, hs)
    hs = rng.choice((32, 64, 64, 128))
    heads = rng.randint(2, 768 // hs)
    layers = rng.randint(2, 8)
    vocab = rng.choice((65, 96, _log_int(rng, 256, 16384)))
    if kind == "generate":
        return generate(layers, heads, hs, _log_int(rng, 1, 16), _size(rng, 64, 512), vocab, _log_int(rng, 16, 128))
    T = _size(rng, 64, 1024)
    return train(rng.choice(("fp32", "tf32")), layers, heads, hs, max(1, min(16, _log_int(rng, 1024, 8192) // T)), T, vocab,
                 rng.randint(2, 4))


# ---- inputs -----------------------------------------------------------------------------------------------------

def _model(case, seed):
    C = case["heads"] * case["hs"]
    padded = -(-case["vocab"] // 128) * 128              # the driver program's padding
    return bmb.Trainer(seed=seed % (1 << 31), max_seq_len=case["T"], vocab_size=case["vocab"], padded_vocab=padded,
                       n_layer=case["layers"], n_head=case["heads"], n_embd=C, B=case["B"], T=case["T"], use_flash=1,
                       math=MATH[case["math"]], fused=1 if case["math"] == "tf32" else 0)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")              # noqa: E731
    uniform = lambda *shape: torch.rand(shape, generator=g, device="cuda") * 2 - 1      # noqa: E731
    empty = lambda *shape: torch.empty(shape, device="cuda")                            # noqa: E731
    s = {"case": case}
    if case["kind"] == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        s["A"], s["B"] = uniform(*((K, M) if case["ta"] else (M, K))), uniform(*((N, K) if case["tb"] else (K, N)))
        s["C"] = uniform(M, N)
    elif case["kind"] == "bgemm":
        n, T, hs = case["batch"], case["T"], case["hs"]
        s["q"], s["k"], s["v"] = normal(n, T, hs), normal(n, T, hs), normal(n, T, hs)
        s["p"] = torch.softmax(normal(n, T, T), dim=-1)                       # weights as the softmax leaves them
        s["scores"], s["out"] = empty(n, T, T), empty(n, T, hs)
    elif case["kind"] == "flash":
        B, T, NH, C = case["B"], case["T"], case["NH"], case["NH"] * case["hs"]
        s["qkv"], s["dout"] = normal(B, T, 3 * C), normal(B, T, C)
        s["out"], s["lse"], s["dsum"], s["dqkv"] = empty(B, T, C), empty(B, NH, T), empty(B, NH, T), empty(B, T, 3 * C)
    elif case["kind"] == "train":
        n = (case["steps"], case["B"], case["T"])
        r = np.random.default_rng(seed)
        pinned = lambda a: torch.from_numpy(a.astype(np.int32)).pin_memory()            # noqa: E731
        s["tokens"], s["targets"] = pinned(r.integers(0, case["vocab"], n)), pinned(r.integers(0, case["vocab"], n))
        s["trainer"] = _model(case, seed)
        s["losses"] = torch.zeros(case["steps"]).pin_memory()
        s["params"] = torch.empty(s["trainer"].num_params).pin_memory()
        s["done"] = 0
    else:
        t = s["trainer"] = _model(case, seed)
        w = torch.empty(t.num_params)
        t.get_params(w)
        # Random weights of the initial size give every token the same chance; three times as large they tell the
        # tokens apart about as much as a trained character model does.
        t.set_params(w * 3)
        s["probs"] = torch.empty(t.cfg.padded_vocab)
        s["seed"] = seed % (1 << 31)
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        if not case["ta"] and not case["tb"]:
            bmb.call(REGISTRY[case["math"]], M, N, K, 1.0, s["A"], s["B"], case["beta"], s["C"])
        else:
            bmb.call("bmb_gemm_ex", MATH[case["math"]], 0, case["ta"], case["tb"], M, N, K, 1.0, s["A"], s["B"], case["beta"], s["C"], None)
        return s["C"]
    if case["kind"] == "bgemm":
        n, T, hs = case["batch"], case["T"], case["hs"]
        bmb.lib().bmb_set_math_mode(MATH[case["math"]])
        bmb.call("bmb_batched_gemm", 0, 1, n, T, T, hs, 1.0 / math.sqrt(hs), s["q"], T * hs, s["k"], T * hs, 0.0, s["scores"], T * T, None)
        bmb.call("bmb_batched_gemm", 0, 0, n, T, hs, T, 1.0, s["p"], T * T, s["v"], T * hs, 0.0, s["out"], T * hs, None)
        return s["scores"], s["out"]
    if case["kind"] == "flash":
        B, T, NH, C = case["B"], case["T"], case["NH"], case["NH"] * case["hs"]
        bmb.lib().bmb_set_math_mode(MATH[case["math"]])
        bmb.call("bmb_flash_attention_forward", s["out"], s["lse"], s["qkv"], B, T, C, NH)
        bmb.call("bmb_flash_attention_backward", s["dqkv"], s["dsum"], s["dout"], s["qkv"], s["out"], s["lse"], B, T, C, NH)
        return s["out"], s["lse"], s["dqkv"]
    t = s["trainer"]
    if case["kind"] == "train":
        for k in range(case["steps"]):
            t.upload(s["tokens"][k], s["targets"][k])
            s["done"] += 1
            t.step(3e-4, s["done"])
            t.loss_async(s["losses"][k:])
        t.get_params(s["params"])
        return s["losses"], s["params"]
    text = t.generate(0, case["tokens"], s["seed"], 0.8)
    window = (([0] + text)[-case["T"]:] + [0] * case["T"])[:case["T"]]
    context = np.zeros((case["B"], case["T"]), dtype=np.int32)
    context[0] = window
    last = min(case["T"], case["tokens"] + 1) - 1
    bmb.call("bmb_trainer_next_token_probs", t.h, context, last, s["probs"])
    return np.asarray(text, dtype=np.int32), s["probs"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def _params(case):
    C = case["heads"] * case["hs"]
    padded = -(-case["vocab"] // 128) * 128
    matmul = case["layers"] * 12 * C * C + padded * C                       # weights that a token is multiplied with
    return matmul, matmul + case["T"] * C + case["layers"] * 13 * C + 2 * C


def work(case):
    if case["kind"] == "gemm":
        M, N, K = case["M"], case["N"], case["K"]
        return {"bytes": 4 * (M * K + K * N + M * N * (2 if case["beta"] else 1)), "flops": 2 * M * N * K}
    if case["kind"] == "bgemm":
        n, T, hs = case["batch"], case["T"], case["hs"]
        return {"bytes": 4 * n * (2 * T * T + 4 * T * hs), "flops": 4 * n * T * T * hs}
    if case["kind"] == "flash":
        B, T, NH, hs = case["B"], case["T"], case["NH"], case["hs"]
        forward = 4 * B * NH * hs * T * (T + 1) // 2
        return {"bytes": 4 * B * T * NH * (8 * hs + 1), "flops": forward + forward * 5 // 2}
    matmul, total = _params(case)
    C, L, T = case["heads"] * case["hs"], case["layers"], case["T"]
    if case["kind"] == "train":
        tokens = case["B"] * T
        attention = 4 * L * tokens * C * (T + 1) // 2
        # per step the weights are read, and the weights and both moments read and written by the optimiser
        return {"bytes": case["steps"] * 4 * 7 * total + 4 * total,
                "flops": case["steps"] * (6 * matmul * tokens + attention * 7 // 2)}
    n = case["tokens"]
    full = max(0, n - T)          # draws from a full window: every position has moved, so the window is computed anew
    grown = n - full
    flops = 2 * matmul * grown + 4 * L * C * grown * (grown + 1) // 2
    flops += (full + 1) * (2 * L * 12 * C * C * min(T, n + 1) + 4 * L * C * T * (T + 1) // 2)
    return {"bytes": 4 * matmul * (n + 1), "flops": flops}


# ---- how far two correct implementations may be apart ----------------------------------------------------------

def tolerance(case):
    # About four times what was measured on B200 over the listed sizes and some drawn ones: products and attention
    # against the same computation in 64 bits (worst seen: fp32 products 1.4e-6 at K = 6144, TF32 2.9e-4, BF16 2.1e-3;
    # attention 9.4e-7 in fp32, 4.8e-4 in TF32; the largest single difference is of a small gradient entry), training
    # against the same steps with the sequences of each batch in another order (6e-7 in fp32, 3.6e-4 in TF32: an AdamW
    # step of an entry whose gradient is all rounding has either sign) -- with some room in fp32, where that order
    # leaves the sums inside a sequence as they were.
    fp32 = case["math"] == "fp32"
    if case["kind"] == "gemm":
        return {"fp32": {"rel": 6e-6, "max": 4e-5}, "tf32": {"rel": 1.2e-3, "max": 8e-3}, "bf16": {"rel": 8.4e-3, "max": 4.6e-2}}[case["math"]]
    if case["kind"] == "bgemm":
        return {"rel": 4e-6, "max": 4e-5} if fp32 else {"rel": 1.2e-3, "max": 1e-2}
    if case["kind"] == "flash":
        return {"rel": 4e-6, "max": 6e-5} if fp32 else {"rel": 2e-3, "max": 5e-2}
    if case["kind"] == "train":
        return {"rel": 5e-6, "max": 1e-2} if fp32 else {"rel": 1.5e-3, "max": 0.22}
    return {"rel": 5e-5, "max": 5e-4}


# ---- the same numbers in 64 bits, from plain torch --------------------------------------------------------------

def exact(case, seed):
    """What run() returns, in 64 bits; None for training and sampling, whose weights the library itself draws."""
    if case["kind"] not in ("gemm", "bgemm", "flash"):
        return None
    s = prepare(case, seed)
    if case["kind"] == "gemm":
        A, B = s["A"].double(), s["B"].double()
        return (A.T if case["ta"] else A) @ (B.T if case["tb"] else B) + case["beta"] * s["C"].double()
    if case["kind"] == "bgemm":
        scores = s["q"].double() @ s["k"].double().transpose(1, 2) / math.sqrt(case["hs"])
        return scores, s["p"].double() @ s["v"].double()
    B, T, NH, hs = case["B"], case["T"], case["NH"], case["hs"]
    heads = lambda x: x.reshape(B, T, NH, hs).transpose(1, 2)                           # noqa: E731
    rows = lambda x: x.transpose(1, 2).reshape(B, T, NH * hs)                           # noqa: E731
    q, k, v = (heads(x) for x in s["qkv"].double().chunk(3, dim=-1))
    dout = heads(s["dout"].double())
    scores = q @ k.transpose(2, 3) / math.sqrt(hs)
    scores.masked_fill_(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), -math.inf)
    lse = torch.logsumexp(scores, dim=-1)
    p = torch.exp(scores - lse[..., None])
    out = p @ v
    dp = dout @ v.transpose(2, 3)
    ds = p * (dp - (dout * out).sum(-1, keepdim=True)) / math.sqrt(hs)
    return rows(out), lse, torch.cat([rows(ds @ k), rows(ds.transpose(2, 3) @ q), rows(p.transpose(2, 3) @ dout)], dim=-1)
