"""Workloads of the package's public entry points, for timing and for comparing the outputs of two builds.

Five kinds of call, each what some program built on this package does over and over:

  attention   ``forgetting_attention`` with its backward (a training step's share of one layer) or without (a prompt
              chunk against the keys so far)
  decode      ``forgetting_attention`` with one query row per sequence against an ``FgateCache``
  block       ``FoxProBlock`` forward and backward: the attention and every operator around it, weights' gradients too
  generate    one token through a stack of ``FoxProBlock`` on an ``FgateCache``
  loss        ``FusedCrossEntropyLoss`` forward and backward over vocabulary logits
"""
import math

import torch
import torch.nn.functional as F

import forgetting_transformer_b200 as fox

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one layer of the smallest training shape the package quotes: a step here is launches and host work
        dict(name="train_b4_t512_h12_d64", kind="attention", train=True, B=4, H=12, M=512, N=512, D=64, dtype="bf16",
             mu=0.0, sigma=1.0, std=1.0, padded=False, threshold="none", head_first=False),
        # fewer queries than keys, lengths that fill no tile, left padding, a fixed pruning threshold, fp16
        dict(name="train_ragged_fp16", kind="attention", train=True, B=4, H=2, M=1020, N=2098, D=64, dtype="fp16",
             mu=2.5, sigma=1.5, std=0.5, padded=True, threshold="-10", head_first=True),
        # the long-context training shape (head dim 64, gates near 1, left padding): the benchmark's default
        dict(name="train_t16384_h24_d64", kind="attention", train=True, B=2, H=24, M=16384, N=16384, D=64,
             dtype="bf16", mu=4.0, sigma=1.0, std=1.0, padded=True, threshold="none", head_first=True),
        # the largest: long context at head dim 128, nothing pruned
        dict(name="train_t16384_h16_d128", kind="attention", train=True, B=4, H=16, M=16384, N=16384, D=128,
             dtype="bf16", mu=-1.0, sigma=1.5, std=1.0, padded=False, threshold="none", head_first=True),
        # the same with strong decay and the automatic threshold: nearly all blocks are skipped
        dict(name="train_pruned_d128", kind="attention", train=True, B=4, H=16, M=16384, N=16384, D=128,
             dtype="bf16", mu=-1.0, sigma=1.5, std=1.0, padded=False, threshold="auto", head_first=True),
        # a chunk of a long prompt against what is already in the cache, no gradients
        dict(name="prefill_chunk_d64", kind="attention", train=False, B=1, H=24, M=3000, N=11000, D=64, dtype="bf16",
             mu=4.0, sigma=1.0, std=1.0, padded=False, threshold="none", head_first=True),
        # serving: a batch of sequences of one odd length, one new token each
        dict(name="decode_b16_n4099_d128", kind="decode", B=16, H=16, N=4099, D=128, dtype="bf16", mu=3.0, sigma=1.0,
             padded=True),
        # one very long sequence, one new token
        dict(name="decode_b1_n65536_d64", kind="decode", B=1, H=24, N=65536, D=64, dtype="bf16", mu=5.0, sigma=1.0,
             padded=False),
        # a layer of the long-context model, one micro-batch
        dict(name="block_train_t16384", kind="block", B=1, T=16384, hidden=1536, heads=24, inter=4096, dtype="bf16",
             padded=False),
        # a layer of a small model on short sequences with left padding
        dict(name="block_train_b4_t512", kind="block", B=4, T=512, hidden=768, heads=12, inter=2048, dtype="bf16",
             padded=True),
        # generation: a token through four layers, two thousand tokens in the cache
        dict(name="generate_n2000", kind="generate", B=1, N=2000, hidden=1536, heads=24, inter=4096, layers=4,
             dtype="bf16", padded=False),
        # the language-model loss of one micro-batch
        dict(name="loss_8192x50304", kind="loss", rows=8192, classes=50304, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# (query, key) pairs times head dim of the largest listed case
MOST_PAIRS = 4 * 16 * 16384 * 16384 // 2 * 128


def draw(rng):
    kind = rng.choices(("train", "infer", "decode", "block", "generate", "loss"), (4, 2, 2, 2, 1, 1))[0]
    if kind in ("train", "infer"):
        N = _log(rng, 128, 16384)
        M = N if rng.random() < 0.6 else max(2, int(N * rng.uniform(0.1, 1.0)))
        D = rng.choice((16, 32, 64, 64, 64, 128, 128, 128))
        H, B = rng.choice((2, 4, 7, 12, 16, 24)), rng.choice((1, 2, 3, 4, 8))
        while B * H * M * N // 2 * D > MOST_PAIRS or B * N > 65536:
            B, H = max(1, B // 2), max(2, H * 3 // 4)
        pruned = rng.random() < 0.35
        return dict(kind="attention", train=kind == "train", B=B, H=H, M=M, N=N, D=D,
                    dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")), mu=rng.uniform(-1, 1) if pruned else rng.uniform(0, 5),
                    sigma=rng.uniform(0.8, 1.5), std=rng.uniform(0.5, 1.0), padded=rng.random() < 0.4,
                    threshold=rng.choice(("auto", "-10")) if pruned else "none", head_first=rng.random() < 0.5)
    if kind == "decode":
        N = _log(rng, 64, 65536)
        B, H = _log(rng, 1, 32), rng.choice((4, 12, 16, 24))
        while B * N > 131072:
            B //= 2
        return dict(kind="decode", B=B, H=H, N=N, D=rng.choice((64, 128)), dtype=rng.choice(("bf16", "bf16", "fp16")),
                    mu=rng.uniform(2, 5), sigma=rng.uniform(0.8, 1.5), padded=rng.random() < 0.4)
    hidden, heads, inter = rng.choice(((512, 8, 1408), (768, 12, 2048), (1024, 16, 2816), (1536, 24, 4096), (2048, 16, 5632)))
    if kind == "block":
        T, B = _log(rng, 64, 16384), rng.choice((1, 2, 4))
        while B * T > 16384:
            B //= 2
        return dict(kind="block", B=B, T=T, hidden=hidden, heads=heads, inter=inter,
                    dtype=rng.choice(("bf16", "bf16", "fp16")), padded=rng.random() < 0.3)
    if kind == "generate":
        return dict(kind="generate", B=_log(rng, 1, 16), N=_log(rng, 64, 8192), hidden=hidden, heads=heads, inter=inter,
                    layers=rng.choice((1, 2, 4)), dtype="bf16", padded=rng.random() < 0.3)
    return dict(kind="loss", rows=_log(rng, 256, 8192), classes=rng.randint(16000, 50304),
                dtype=rng.choice(("bf16", "bf16", "fp32")))


# ---------------------------------------------------------------- inputs

def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)


def _seq_start(gen, case, length):
    """First valid position of each sequence: left padding of up to an eighth of the length."""
    if not case["padded"]:
        return None
    return torch.randint(0, max(1, length // 8), (case["B"],), generator=gen, device="cuda")


def _mask(gen, case, length):
    start = _seq_start(gen, case, length)
    if start is None:
        return None
    return (torch.arange(length, device="cuda")[None, :] >= start[:, None]).long()


def _block(case):
    """A layer with norm weights away from 1, as after training."""
    blk = fox.FoxProBlock(case["hidden"], case["heads"], case["inter"], fgate_bias=5.0).cuda().to(DTYPES[case["dtype"]])
    with torch.no_grad():
        for m in (blk.attn_norm, blk.mlp_norm, blk.attn.q_norm, blk.attn.k_norm, blk.attn.output_norm):
            m.weight.uniform_(0.5, 1.5)
    return blk


def _prepare_attention(case, gen):
    B, H, M, N, D, dt = (case[k] for k in ("B", "H", "M", "N", "D", "dtype"))
    dt = DTYPES[dt]
    q, k, v = (_randn(gen, B, H, t, D) * case["std"] for t in (M, N, N))
    if case["threshold"] == "auto":     # heads of different scales, so that their thresholds differ
        scale = torch.rand(H, generator=gen, device="cuda")[None, :, None, None] * 1.5 + 0.5
        q, k, v = q * scale, k * scale, v * scale
    gate = F.logsigmoid(_randn(gen, B, H, N) * case["sigma"] + case["mu"])
    dout = _randn(gen, B, H, M, D)
    if not case["head_first"]:
        q, k, v, dout = (t.transpose(1, 2).contiguous() for t in (q, k, v, dout))
        gate = gate.transpose(1, 2).contiguous()
    q, k, v, dout = (t.to(dt) for t in (q, k, v, dout))
    state = dict(case=case, inputs=[t.requires_grad_(case["train"]) for t in (q, k, v, gate)],
                 seq_start=_seq_start(gen, case, N))
    if case["train"]:
        state["dout"] = dout
    state["threshold"] = {"none": None, "auto": "auto"}.get(case["threshold"], case["threshold"])
    if state["threshold"] not in (None, "auto"):
        state["threshold"] = float(state["threshold"])
    return state


def _prepare_decode(case, gen):
    B, H, N, D, dt = case["B"], case["H"], case["N"], case["D"], DTYPES[case["dtype"]]
    cache = fox.FgateCache()
    cache.update(_randn(gen, B, H, N, D, dtype=dt), _randn(gen, B, H, N, D, dtype=dt),
                 F.logsigmoid(_randn(gen, B, H, N) * case["sigma"] + case["mu"]), 0)
    return dict(case=case, cache=cache, q=_randn(gen, B, H, 1, D, dtype=dt), seq_start=_seq_start(gen, case, N))


def _prepare_block(case, gen):
    B, T, C, dt = case["B"], case["T"], case["hidden"], DTYPES[case["dtype"]]
    blk = _block(case)
    return dict(case=case, block=blk, params=list(blk.parameters()), x=_randn(gen, B, T, C, dtype=dt).requires_grad_(),
                dout=_randn(gen, B, T, C, dtype=dt), mask=_mask(gen, case, T))


def _prepare_generate(case, gen):
    B, N, C, H, dt = case["B"], case["N"], case["hidden"], case["heads"], DTYPES[case["dtype"]]
    cache = fox.FgateCache()
    blocks = [_block(case) for _ in range(case["layers"])]
    for i, blk in enumerate(blocks):
        st = blk.attn.init_shift_state(B)
        for s in st.values():
            s.copy_(_randn(gen, B, C))
        cache.update_shift_cache(st["key_shift"], st["value_shift"], i)
        cache.update(_randn(gen, B, H, N, C // H, dtype=dt), _randn(gen, B, H, N, C // H, dtype=dt),
                     F.logsigmoid(_randn(gen, B, H, N) + 5.0), i)
    return dict(case=case, blocks=blocks, cache=cache, x=_randn(gen, B, 1, C, dtype=dt), mask=_mask(gen, case, N + 1))


def _prepare_loss(case, gen):
    rows, classes = case["rows"], case["classes"]
    dt = torch.float32 if case["dtype"] == "fp32" else DTYPES[case["dtype"]]
    logits = torch.empty(rows, classes, dtype=dt, device="cuda").normal_(0.0, 2.0, generator=gen).requires_grad_()
    labels = torch.randint(0, classes, (rows,), generator=gen, device="cuda")
    labels[::7] = -100      # positions without a target
    return dict(case=case, loss=fox.FusedCrossEntropyLoss(), logits=logits, labels=labels)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)     # module initialisation draws from the default generators
    return {"attention": _prepare_attention, "decode": _prepare_decode, "block": _prepare_block,
            "generate": _prepare_generate, "loss": _prepare_loss}[case["kind"]](case, gen)


# ---------------------------------------------------------------- one pass

def _run_attention(s):
    case, inputs = s["case"], s["inputs"]
    if not case["train"]:
        with torch.no_grad():
            return fox.forgetting_attention(*inputs, head_first=case["head_first"], seq_start=s["seq_start"],
                                            adaptive_threshold=s["threshold"])
    for t in inputs:
        t.grad = None
    out = fox.forgetting_attention(*inputs, head_first=case["head_first"], seq_start=s["seq_start"],
                                   adaptive_threshold=s["threshold"])
    out.backward(s["dout"])
    return [out] + [t.grad for t in inputs]


def _run_decode(s):
    with torch.no_grad():
        return fox.forgetting_attention(s["q"], *s["cache"][0], head_first=True, seq_start=s["seq_start"])


def _run_block(s):
    s["x"].grad = None
    for p in s["params"]:
        p.grad = None
    out = s["block"](s["x"], s["mask"])
    out.backward(s["dout"])
    return [out, s["x"].grad] + [p.grad for p in s["params"]]


def _run_generate(s):
    cache = s["cache"]
    cache.crop(s["case"]["N"])      # back to the prompt: the next candidate for the same position
    with torch.no_grad():
        h = s["x"]
        for i, blk in enumerate(s["blocks"]):
            h = blk(h, s["mask"], cache, i)
    return [h, cache.to_legacy_cache(), cache.key_shift_cache, cache.value_shift_cache]


def _run_loss(s):
    s["logits"].grad = None
    loss = s["loss"](s["logits"], s["labels"])
    loss.backward()
    return [loss, s["logits"].grad]


_RUN = {"attention": _run_attention, "decode": _run_decode, "block": _run_block, "generate": _run_generate,
        "loss": _run_loss}


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ---------------------------------------------------------------- what a pass cannot do without

def _pairs(M, N):
    """(query, key) pairs of the causal triangle whose last row sees all N keys."""
    return M * (N - M) + M * (M + 1) / 2


def work(case):
    kind = case["kind"]
    if kind == "attention":
        B, H, M, N, D = (case[k] for k in ("B", "H", "M", "N", "D"))
        pairs = _pairs(M, N)
        if case["threshold"] != "none":     # about two key blocks of 128 per query row are left at these decays
            pairs = min(pairs, 256.0 * M)
        rows, gates = B * H * (2 * M + 2 * N) * D * 2, B * H * N * 4    # q, out, k, v; gates
        if case["train"]:                   # and dout, dq, dk, dv; gate gradients
            return dict(bytes=2 * (rows + gates), flops=14.0 * D * B * H * pairs)
        return dict(bytes=rows + gates, flops=4.0 * D * B * H * pairs)
    if kind == "decode":
        B, H, N, D = (case[k] for k in ("B", "H", "N", "D"))
        return dict(bytes=B * H * (2 * N * D * 2 + 4 * N + 4 * D), flops=4.0 * B * H * N * D)
    if kind == "loss":
        n = case["rows"] * case["classes"] * (4 if case["dtype"] == "fp32" else 2)
        return dict(bytes=2 * n + 8 * case["rows"], flops=0)
    C, H, inter = case["hidden"], case["heads"], case["inter"]
    weights = 5 * C * C + 3 * C * inter + 3 * C * H
    if kind == "block":
        tokens = case["B"] * case["T"]
        return dict(bytes=2 * (4 * tokens * C + 2 * weights),
                    flops=6.0 * tokens * weights + 14.0 * C * case["B"] * _pairs(case["T"], case["T"]))
    B, N, layers = case["B"], case["N"], case["layers"]
    return dict(bytes=layers * (2 * weights + B * (4 * N * C + 4 * H * N)) + 4 * B * C,
                flops=layers * B * (2.0 * weights + 4.0 * N * C))


def tolerance(case):
    # results are rounded to 16 bits, and products take 16-bit operands (probabilities and their gradients among
    # them, rounded at points that implementations choose differently); sums and exponents are fp32
    if case["kind"] == "loss":      # fp32 loss, gradient rounded once to the logits' type
        return dict(rel=1e-5 if case["dtype"] == "fp32" else 3e-3, max=1e-3 if case["dtype"] == "fp32" else 2e-2)
    if case["kind"] in ("block", "generate"):   # a chain of such results
        return dict(rel=2e-2 if case["dtype"] == "bf16" else 4e-3)
    return dict(rel=1e-2 if case["dtype"] == "bf16" else 2e-3)
