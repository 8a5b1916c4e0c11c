"""Performance cases: what programs built on this framework have it do, through its public entry points.

Every program family of the framework is here once or more, at the sizes of its benchmark
configurations, and `draw` spreads the same families over the sizes, data types and options that the
entry points take in earnest: batches from a few sequences to the full one, odd and ragged sizes,
hidden widths between and at the configured ones.  A case's "op" names the family:

    stacked    ops.lstm_stacked                 rectangular batch, packed weights kept by the caller
    words      frontend.embed -> stacked_lstm -> project_softmax on a ragged batch of word ids
    dilated    ops.lstm_dilated
    grid       ops.grid_rnn
    b2b        ops.b2b_gemm
    attention  ops.flash_attention              full, causal, sliding and two-sided windows
    sparse     ops.sparse_attention
    rnn_attn   ops.rnn_attention                encoder, attention and decoder on padded ragged batches
"""
import math
import random

import torch

from fractaltensor_b200 import frontend, ops

_DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # The smallest configured model, fp32, one small batch: a chain of 67 tiny dependent levels.
        {"name": "stacked fp32 small", "op": "stacked", "dtype": "f32", "D": 4, "L": 64, "N": 32, "H": 256},
        # An ordinary model: 8 layers of 512, a batch of 64, 100 steps.
        {"name": "stacked fp16 ordinary", "op": "stacked", "dtype": "f16", "D": 8, "L": 100, "N": 64, "H": 512},
        # The largest configured model: 16 layers of 1024 at the full batch of 256.
        {"name": "stacked bf16 large", "op": "stacked", "dtype": "bf16", "D": 16, "L": 100, "N": 256, "H": 1024},
        # A word-level language model as a script writes it: word ids of sentences of different
        # lengths in, next-word probabilities out, parameters handed over unpacked as in training.
        {"name": "words ragged bf16", "op": "words", "dtype": "bf16", "D": 3, "L": 60, "N": 64, "H": 512, "V": 10000},
        # Dilated LSTM, six layers of 256, dilations 1..32, long sequences.
        {"name": "dilated fp16", "op": "dilated", "dtype": "f16", "D": 6, "L": 512, "N": 256, "H": 256},
        # Grid RNN over two sentences of 32 words each.
        {"name": "grid fp16", "op": "grid", "dtype": "f16", "D": 1, "A": 32, "B": 32, "N": 64, "H": 256},
        # Back-to-back GEMM at the smaller sizes of the reference's benchmark: latency and launch cost.
        {"name": "b2b fp16 small", "op": "b2b", "dtype": "f16", "batch": 1, "M": 8192, "n": 256, "K": 64, "P": 64},
        # The same at the configured size: memory-bound.
        {"name": "b2b fp16 large", "op": "b2b", "dtype": "f16", "batch": 16, "M": 16384, "n": 128, "K": 128, "P": 128},
        # Attention of a training-sized batch, full walk.
        {"name": "attention fp16 full", "op": "attention", "dtype": "f16", "mode": "full", "B": 16, "heads": 16,
         "S": 2048, "left": 0, "right": 0},
        # Prefill of one sequence, causal.
        {"name": "attention bf16 causal", "op": "attention", "dtype": "bf16", "mode": "causal", "B": 1, "heads": 16,
         "S": 2048, "left": 0, "right": 0},
        # Token-level sparse attention at the sizes its example gives: window, random and global keys.
        {"name": "sparse fp32", "op": "sparse", "dtype": "f32", "B": 2, "heads": 16, "S": 4096, "d": 64, "window": 5,
         "dilation": 2, "n_global": 3, "R": 3},
        # Attention RNN (encoder, attention, decoder) on sentence pairs of different lengths.
        {"name": "rnn_attn bf16", "op": "rnn_attn", "dtype": "bf16", "Ls": 50, "Lt": 50, "N": 64, "H": 512},
    ]


# ------------------------------------------------------------------------------- more of the same ranges
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _most_flops():
    return work(listed()[2])["flops"]


def draw(rng):
    largest = _most_flops()
    while True:
        c = _draw_any(rng)
        w = work(c)
        # a chain of dependent steps costs time beyond its arithmetic: at most the largest case's
        # operations, and for the memory-bound ones a few times the largest listed bytes
        if w["flops"] <= largest and w["bytes"] <= 1.2e9:
            return c


def _draw_any(rng):
    op = rng.choice(["stacked", "stacked", "words", "dilated", "grid", "b2b", "attention", "attention", "sparse",
                     "rnn_attn"])
    half = rng.choice(["f16", "bf16"])
    if op == "stacked":
        if rng.random() < 0.25:
            return {"op": op, "dtype": "f32", "D": rng.randint(1, 4), "L": rng.randint(16, 100),
                    "N": _log_int(rng, 1, 64), "H": rng.choice([64, 128, 192, 256])}
        return {"op": op, "dtype": half, "D": rng.randint(1, 16), "L": rng.randint(16, 128), "N": _log_int(rng, 1, 256),
                "H": 64 * _log_int(rng, 2, 16)}
    if op == "words":
        return {"op": op, "dtype": half, "D": rng.randint(1, 4), "L": rng.randint(20, 100), "N": _log_int(rng, 4, 128),
                "H": rng.choice([256, 512, 640]), "V": _log_int(rng, 2000, 12000)}
    if op == "dilated":
        return {"op": op, "dtype": half, "D": rng.randint(3, 6), "L": rng.randint(64, 512), "N": _log_int(rng, 8, 256),
                "H": rng.choice([64, 128, 256])}
    if op == "grid":
        return {"op": op, "dtype": half, "D": rng.randint(1, 3), "A": rng.randint(6, 40), "B": rng.randint(6, 40),
                "N": _log_int(rng, 4, 64), "H": rng.choice([64, 128, 256])}
    if op == "b2b":
        K, P = rng.choice([64, 128]), rng.choice([64, 128])
        return {"op": op, "dtype": half, "batch": _log_int(rng, 1, 16), "M": 128 * _log_int(rng, 4, 128),
                "n": rng.choice([128, 256, 512] if K + P < 256 else [128, 256]), "K": K, "P": P}
    if op == "attention":
        mode = rng.choice(["full", "causal", "window", "local"])
        S = 256 * _log_int(rng, 1, 16)
        return {"op": op, "dtype": half, "mode": mode, "B": _log_int(rng, 1, 16), "heads": rng.randint(4, 16), "S": S,
                "left": _log_int(rng, 32, S) if mode in ("window", "local") else 0,
                "right": _log_int(rng, 32, S) if mode == "local" else 0}
    if op == "sparse":
        return {"op": op, "dtype": rng.choice(["f32", "f16", "bf16"]), "B": _log_int(rng, 1, 8),
                "heads": rng.randint(4, 16), "S": _log_int(rng, 256, 8192), "d": rng.choice([32, 64, 128]),
                "window": rng.choice([3, 5, 7]), "dilation": rng.randint(1, 3), "n_global": rng.randint(1, 4),
                "R": rng.randint(1, 4)}
    return {"op": op, "dtype": half, "Ls": rng.randint(8, 64), "Lt": rng.randint(8, 64), "N": _log_int(rng, 2, 128),
            "H": rng.choice([128, 256, 512])}


# ---------------------------------------------------------------------------------------------- inputs
def _lengths(n, longest):
    """n sentence lengths spread evenly over 1/6 .. 1 of the longest, as plain integers."""
    low = max(1, longest // 6)
    return [longest] if n == 1 else [low + (longest - low) * i // (n - 1) for i in range(n)]


def _uniform(g, bound, dt, *shape):
    return ((torch.rand(*shape, device="cuda", generator=g) * 2 - 1) * bound).to(dt)


def _normal(g, scale, dt, *shape):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dt)


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    op = case["op"]
    st = {"case": case}
    if op in ("stacked", "dilated"):
        D, L, N, H = case["D"], case["L"], case["N"], case["H"]
        bound = 1.0 / math.sqrt(H)
        st["x"] = _normal(g, 1.0, dt, L, N, H)
        st["Wp"], st["bias"] = ops.lstm_pack_weights(_uniform(g, bound, dt, D, 4, H, H), _uniform(g, bound, dt, D, 4, H, H),
                                                     _uniform(g, bound, dt, D, 4, H))
        st["dilations"] = [2 ** l for l in range(D)]
    elif op == "words":
        D, N, H, V = case["D"], case["N"], case["H"], case["V"]
        bound = 1.0 / math.sqrt(H)
        lens = _lengths(N, case["L"])
        random.Random(seed).shuffle(lens)
        ids = torch.randint(0, V, (sum(lens),), device="cuda", generator=g)
        st["words"] = frontend.FractalTensor(ids, [list(range(n)) for n in lens], (1,))
        st["table"] = _normal(g, 1.0, dt, V, H)
        st["params"] = [frontend.FractalTensor.from_dense(_uniform(g, bound, dt, D, 4, H, H), 2),
                        frontend.FractalTensor.from_dense(_uniform(g, bound, dt, D, 4, H, H), 2),
                        frontend.FractalTensor.from_dense(_uniform(g, bound, dt, D, 4, 1, H), 2)]
        st["proj"] = _normal(g, 0.25, dt, H, V)
    elif op == "grid":
        D, A, B, N, H = case["D"], case["A"], case["B"], case["N"], case["H"]
        bound = 1.0 / 16
        st["X"], st["Y"] = _normal(g, 1.0, dt, A, B, N, H), _normal(g, 1.0, dt, A, B, N, H)
        st["Wpx"], st["Wpy"] = (ops.grid_pack_weights(_uniform(g, bound, dt, D, 2 * H, H), _uniform(g, bound, dt, D, H, H))
                                for _ in range(2))
        st["bx"], st["by"] = (_uniform(g, bound, torch.float32, D, H) for _ in range(2))
    elif op == "b2b":
        batch, M, n, K, P = case["batch"], case["M"], case["n"], case["K"], case["P"]
        st["A"] = _normal(g, 1.0 / math.sqrt(K), dt, batch, M, K)
        st["B"] = _normal(g, 1.0 / math.sqrt(K), dt, batch, n, K)
        st["C"] = _normal(g, 1.0 / math.sqrt(n), dt, batch, P, n)
    elif op == "attention":
        shape = (case["B"], case["heads"], case["S"], 128)
        st["q"], st["k"], st["v"] = (_normal(g, 1.0, dt, *shape) for _ in range(3))
    elif op == "sparse":
        B, heads, S, d = case["B"], case["heads"], case["S"], case["d"]
        st["q"], st["k"], st["v"] = (_normal(g, 1.0, dt, B, heads, S, d) for _ in range(3))
        st["pos"] = torch.randint(0, S, (B, heads, S - 2 * case["n_global"], case["R"]), device="cuda", generator=g,
                                  dtype=torch.int32)
    else:
        Ls, Lt, N, H = case["Ls"], case["Lt"], case["N"], case["H"]
        bound = 1.0 / math.sqrt(H)
        st["src"], st["trg"] = _normal(g, 1.0, dt, Ls, N, H), _normal(g, 1.0, dt, Lt, N, H)
        st["Ws"], st["Wt"] = (ops.rnn_pack_weights(_uniform(g, bound, dt, H, H), _uniform(g, bound, dt, H, H))
                              for _ in range(2))
        st["bs"], st["bt"] = (_uniform(g, bound, torch.float32, H) for _ in range(2))
        st["enc_proj"], st["dec_proj"] = (torch.rand(H, device="cuda", generator=g).to(dt) for _ in range(2))
        lens = _lengths(N, Ls)
        random.Random(seed).shuffle(lens)
        st["lens"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
    return st


# ------------------------------------------------------------------------------------------ one pass
def run(st):
    case = st["case"]
    op = case["op"]
    if op == "stacked":
        return ops.lstm_stacked(st["x"], st["Wp"], st["bias"])
    if op == "words":
        hs = frontend.stacked_lstm(frontend.embed(st["words"], st["table"]), *st["params"])
        return hs.data, frontend.project_softmax(hs, st["proj"]).data
    if op == "dilated":
        # the cell state buffer is the entry point's scratch beyond a layer's own dilation: hidden states only
        return ops.lstm_dilated(st["x"], st["Wp"], st["dilations"], st["bias"])[0]
    if op == "grid":
        return ops.grid_rnn(st["X"], st["Y"], st["Wpx"], st["Wpy"], st["bx"], st["by"])
    if op == "b2b":
        return ops.b2b_gemm(st["A"], st["B"], st["C"])
    if op == "attention":
        scale = 1.0 / math.sqrt(128.0)
        if case["mode"] == "local":
            return ops.flash_attention(st["q"], st["k"], st["v"], scale=scale, local=(case["left"], case["right"]))
        return ops.flash_attention(st["q"], st["k"], st["v"], scale=scale, causal=case["mode"] != "full",
                                   window=case["left"] if case["mode"] == "window" else None)
    if op == "sparse":
        return ops.sparse_attention(st["q"], st["k"], st["v"], st["pos"], window_size=case["window"],
                                    dilation=case["dilation"], n_global=case["n_global"],
                                    scale=1.0 / math.sqrt(case["d"]))
    return ops.rnn_attention(st["src"], st["trg"], st["Ws"], st["Wt"], st["bs"], st["bt"], st["enc_proj"],
                             st["dec_proj"], st["lens"])


# --------------------------------------------------------------------- what a pass cannot do without
def _visible_pairs(case):
    """(query, key) pairs that the mask leaves, per head."""
    S = case["S"]
    if case["mode"] == "full":
        return S * S
    left = {"causal": S, "window": case["left"] - 1, "local": case["left"]}[case["mode"]]
    right = case["right"] if case["mode"] == "local" else 0
    return sum(min(S - 1, i + right) - max(0, i - left) + 1 for i in range(S))


def work(case):
    es = 4 if case["dtype"] == "f32" else 2
    op = case["op"]
    if op in ("stacked", "dilated"):
        D, L, N, H = case["D"], case["L"], case["N"], case["H"]
        state = D * N * H * 4 if op == "stacked" else 0
        return {"bytes": (D * 8 * H * H + L * N * H + D * L * N * H) * es + D * 4 * H * 4 + state,
                "flops": 16.0 * D * L * N * H * H}
    if op == "words":
        D, H, V = case["D"], case["H"], case["V"]
        T = sum(_lengths(case["N"], case["L"]))
        return {"bytes": T * 8 + (2 * T * H + D * 8 * H * H + H * V) * es + T * V * 4,
                "flops": 16.0 * D * T * H * H + 2.0 * T * H * V}
    if op == "grid":
        D, cells, H = case["D"], case["A"] * case["B"] * case["N"], case["H"]
        return {"bytes": (2 * cells * H + 2 * D * cells * H + 2 * D * 3 * H * H) * es + 2 * D * H * 4,
                "flops": 12.0 * D * cells * H * H}
    if op == "b2b":
        batch, M, n, K, P = case["batch"], case["M"], case["n"], case["K"], case["P"]
        return {"bytes": batch * (M * K + n * K + P * n + M * P) * es, "flops": 2.0 * batch * M * n * (K + P)}
    if op == "attention":
        bh = case["B"] * case["heads"]
        return {"bytes": 4 * bh * case["S"] * 128 * es, "flops": 4.0 * bh * _visible_pairs(case) * 128}
    if op == "sparse":
        bh, S, d, ng = case["B"] * case["heads"], case["S"], case["d"], case["n_global"]
        keys = (S - 2 * ng) * (case["window"] + case["R"]) + 4 * ng * ng
        return {"bytes": 4 * bh * S * d * es + bh * (S - 2 * ng) * case["R"] * 4, "flops": 4.0 * bh * keys * d}
    Ls, Lt, N, H = case["Ls"], case["Lt"], case["N"], case["H"]
    pairs = Lt * sum(_lengths(N, Ls))
    return {"bytes": (2 * Ls * N * H + 2 * Lt * N * H + 4 * H * H + 2 * H) * es + N * 4,
            "flops": 4.0 * (Ls + Lt) * N * H * H + 2.0 * (pairs + (Ls + Lt) * N) * H}


def tolerance(case):
    """What one rounding per stored value gives, over a few dependent layers or steps: fp32 sums in
    another order, or 16-bit hidden states with 10 (fp16) or 7 (bf16) stored bits."""
    return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
