"""Workloads of the training-step library, for timing it and for comparing the outputs of two builds.

A case is one call, or one optimizer update, of a program that uses the `ane` package: `train` runs the micro-steps
of one update (Engine.step / step_tokens), `loss` and `logits` evaluate windows of tokens (eval_loss, eval_logits),
`decode` generates with the KV cache (decode_greedy, decode_sample).  Sizes are the ones of the benchmark, of the
parity configuration (dim 288, head size 48) and of the range between them: one window per step, as the Go engine
trains, up to micro-batches of 8192 tokens, window lengths that are no multiple of any tile, grouped heads, and the
three compute types.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "autoresearch-go-ane_b200"))

import ane  # noqa: E402

DTYPES = {"bf16": ane.DTYPE_BF16, "f32": ane.DTYPE_F32, "bf16x3": ane.DTYPE_BF16X3}

#: The three model sizes that llama2.c-style files come in here: dim, hidden, layers, heads (head size 48 or 64).
SMALL = {"dim": 288, "hidden": 768, "layers": 6, "heads": 6, "kv_heads": 6, "vocab": 32000}
MIDDLE = {"dim": 512, "hidden": 1376, "layers": 8, "heads": 8, "kv_heads": 8, "vocab": 32000}
LARGE = {"dim": 768, "hidden": 2048, "layers": 12, "heads": 12, "kv_heads": 12, "vocab": 32000}

#: FLOPs of the largest listed update (the benchmark's step); drawn cases stay below.
MOST_FLOPS = 5.5e12


def _train(name, size, **kw):
    case = {"name": name, "do": "train", "arch": "llama", "dtype": "bf16", "quirks": False, **size, "seq": 256, "batch": 1,
            "accum": 1, "host_batches": False}
    case.update(kw)
    return case


def listed():
    return [
        # The benchmark's step: 32 windows of 256 tokens, one update per step.
        _train("train_110m_32x256", LARGE, batch=32),
        # The Go engine's own step: one window per call, the update after every call.
        _train("train_110m_1x256", LARGE, batch=1),
        # A long-context run with grouped heads.
        _train("train_gqa_8x1024", LARGE, kv_heads=4, seq=1024, batch=8),
        # The network that the Go engine trains (ReLU^2, QK-norm, value embeddings) with exact gradients.
        _train("train_reference_arch_32x256", LARGE, arch="reference", batch=32),
        # A small model on a corpus of short documents: head size 48, windows of 200 tokens, batches from the host,
        # three micro-steps per update.
        _train("train_small_5x200_accum3", SMALL, seq=200, batch=5, accum=3, host_batches=True),
        # The stated fp32 parity configuration.
        _train("train_small_f32_8x256", SMALL, dtype="f32", batch=8),
        # The reference's own step, quirks included, at split precision: the mode that stays within its tolerance.
        _train("train_reference_bf16x3_2x256", LARGE, arch="reference", dtype="bf16x3", quirks=True, batch=2),
        # The evaluation loop of the harness: 64 windows, only the loss comes back.
        {"name": "eval_loss_64x256", "do": "loss", "arch": "llama", "dtype": "bf16", **LARGE, "seq": 256, "batch": 64, "windows": 64},
        # EvalLogits as the harness calls it: one window, a fresh [vocab][seq] array on the host.
        {"name": "eval_logits_1x256", "do": "logits", "arch": "llama", "dtype": "bf16", **LARGE, "seq": 256, "batch": 1, "windows": 1},
        # The smallest evaluation: one ragged window of a small model.
        {"name": "eval_loss_small_1x100", "do": "loss", "arch": "llama", "dtype": "bf16", **SMALL, "seq": 100, "batch": 1, "windows": 1},
        # Batched generation with grouped heads: 32 prompts of 512 tokens, 256 new ones each.
        {"name": "decode_gqa_32x512_256", "do": "decode", "arch": "llama", "dtype": "bf16", **LARGE, "kv_heads": 4, "seq": 1024,
         "batch": 32, "prompt": 512, "new": 256, "temperature": 0.0},
        # One interactive completion: a short prompt, sampled at temperature 0.8.
        {"name": "decode_110m_1x37_64", "do": "decode", "arch": "llama", "dtype": "bf16", **LARGE, "seq": 256, "batch": 1,
         "prompt": 37, "new": 64, "temperature": 0.8},
    ]


# ---- drawn cases ----------------------------------------------------------------------------------------------------
def _between(rng, lo, hi):
    """A whole number from lo to hi, even over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng):
    size = dict(rng.choice([SMALL, MIDDLE, LARGE]))
    size["kv_heads"] = size["heads"] // rng.choice([1, 1, 1, 2, size["heads"] // 2])
    size["vocab"] = rng.choice([32000, 32000, 4096])
    return size


def _seq(rng):
    """Half of the runs use a power of two, the other half whatever the documents are cut into."""
    return rng.choice([128, 256, 512, 1024]) if rng.random() < 0.5 else _between(rng, 48, 1024)


def _fit(case, key, most_flops):
    """Halves `key` until one pass fits."""
    while case[key] > 1 and work(case)["flops"] > most_flops:
        case[key] = (case[key] + 1) // 2
    return case


def draw(rng):
    do = rng.choice(["train"] * 5 + ["loss"] * 2 + ["logits"] + ["decode"] * 3)
    size, seq = _size(rng), _seq(rng)
    if do == "train":
        case = _train("", size, seq=seq, batch=_between(rng, 1, 32), accum=rng.choice([1, 1, 2, 4]), host_batches=rng.random() < 0.5)
        del case["name"]
        case["dtype"] = rng.choice(["bf16"] * 6 + ["f32", "bf16x3"])
        if rng.random() < 0.25:
            case.update(arch="reference", kv_heads=case["heads"])
        if case["dtype"] != "bf16":  # a parity run: a few windows
            case["quirks"] = case["arch"] == "reference"
            case["accum"] = 1
            return _fit(case, "batch", 0.35e12)
        case = _fit(case, "batch", MOST_FLOPS)
        return _fit(case, "accum", MOST_FLOPS)
    case = {"do": do, "arch": "llama", "dtype": "bf16", **size, "seq": seq}
    if do == "loss":
        case.update(batch=_between(rng, 1, 64), windows=_between(rng, 1, 64))
        return _fit(_fit(case, "windows", 3.6e12), "batch", 3.6e12)
    if do == "logits":
        case.update(seq=max(48, min(512, seq // 4 * 4)), batch=1, windows=rng.choice([1, 1, 2, 3]))
        return case
    new = _between(rng, 8, 200)
    prompt = _between(rng, 4, 500)
    case.update(seq=rng.choice([s for s in (256, 512, 1024) if s >= prompt + new]), batch=_between(rng, 1, 32), prompt=prompt, new=new,
                temperature=rng.choice([0.0, 0.0, 0.7, 1.0]))
    return case


# ---- what a user's program has in hand ------------------------------------------------------------------------------
_staging = None  # page-locked memory that weights pass through on their way from the generator to the engine


def _put(engine, tensor_id, layer, values):
    global _staging
    n = values.numel()
    if _staging is None or _staging.numel() < n:
        _staging = torch.empty(n, dtype=torch.float32, pin_memory=True)
    _staging[:n].copy_(values.reshape(-1))
    engine.import_tensor(tensor_id, layer, _staging[:n].numpy())


def _random_weights(engine, case, gen):
    """N(0, 0.02) matrices and the initial lambdas of the reference, as the benchmark sets them."""
    normal = lambda n, std=0.02: torch.randn(n, generator=gen, device="cuda") * std  # noqa: E731
    layered = (ane.T_WQ, ane.T_WK, ane.T_WV, ane.T_WO, ane.T_W1, ane.T_W3, ane.T_W2, ane.T_VE_EMBED)
    for layer in range(case["layers"]):
        for tid in layered:
            n = engine.tensor_size(tid, layer)
            if n > 0:
                _put(engine, tid, layer, normal(n))
        n = engine.tensor_size(ane.T_VE_GATE, layer)
        if n > 0:
            _put(engine, ane.T_VE_GATE, layer, torch.rand(n, generator=gen, device="cuda") * 0.02)
    for tid in (ane.T_EMBED, ane.T_SMEAR_GATE):
        n = engine.tensor_size(tid, 0)
        if n > 0:
            _put(engine, tid, 0, normal(n))
    for tid, value in ((ane.T_X0_LAMBDAS, 0.1), (ane.T_SMEAR_LAMBDA, 0.01), (ane.T_BACKOUT_LAMBDA, 0.01)):
        n = engine.tensor_size(tid, 0)
        if n > 0:
            _put(engine, tid, 0, torch.full((n,), value))


def _successor_weights(engine, case, gen):
    """Weights of a model that is as sure of its next token as a trained one: random weights put the best two of 32000
    logits so close together that rounding picks the winner, and one different token changes everything after it.

    Token v has the embedding [c(v) | c(next(v))] with next a random permutation; the first feed-forward block moves the
    second half to the first (silu(u) u - silu(-u) (-u) = u^2 tanh(u / 2), per component), so that the classifier, which
    is the embedding, finds next(v).  All other weights are random, residual writers scaled down with the depth."""
    _random_weights(engine, case, gen)
    dim, hidden, vocab, layers = case["dim"], case["hidden"], case["vocab"], case["layers"]
    half = dim // 2
    code = torch.randn(vocab, half, generator=gen, device="cuda")
    follows = torch.randperm(vocab, generator=gen, device="cuda")
    _put(engine, ane.T_EMBED, 0, 0.1 * torch.cat([code, code[follows]], 1))
    std = 0.02 / math.sqrt(2 * layers)
    for layer in range(layers):
        _put(engine, ane.T_WO, layer, torch.randn(dim, dim, generator=gen, device="cuda") * std)
        _put(engine, ane.T_W2, layer, torch.randn(dim, hidden, generator=gen, device="cuda") * std)
    at = torch.arange(half, device="cuda")
    w1 = torch.randn(hidden, dim, generator=gen, device="cuda") * 0.02
    w1[:dim] = 0
    w1[at, half + at] = 1.0
    w1[half + at, half + at] = -1.0
    w2 = torch.randn(dim, hidden, generator=gen, device="cuda") * std
    w2[:, :dim] = 0
    w2[at, at] = 1.0
    w2[at, half + at] = -1.0
    _put(engine, ane.T_W1, 0, w1)
    _put(engine, ane.T_W3, 0, w1)
    _put(engine, ane.T_W2, 0, w2)


def _zipf_tokens(n, vocab, rng):
    """Token ids of natural text: i.i.d. Zipf(1.1)."""
    cdf = np.cumsum(np.arange(1, vocab + 1, dtype=np.float64) ** -1.1)
    return np.minimum(np.searchsorted(cdf, rng.random(n) * cdf[-1], side="right"), vocab - 1).astype(np.uint16)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    train = case["do"] == "train"
    seq = case["seq"]
    stream = _zipf_tokens(1 << 16, case["vocab"], rng)
    engine = ane.open(ane.Options(
        tokens=stream if train else None, dim=case["dim"], hidden=case["hidden"], n_layers=case["layers"], n_heads=case["heads"],
        n_kv_heads=case["kv_heads"], vocab=case["vocab"], seq=seq, batch=case["batch"], seed=1 + seed % 1000003,
        arch=ane.ARCH_REFERENCE if case["arch"] == "reference" else ane.ARCH_LLAMA, quirks=int(case.get("quirks", False)),
        compute_dtype=DTYPES[case["dtype"]], accum_steps=case.get("accum", 1), lr=3e-4, adam_beta1=0.9, adam_beta2=0.95,
        weight_decay=0.1, grad_clip=1.0))
    state = {"case": case, "engine": engine}
    if case["do"] == "decode":
        _successor_weights(engine, case, gen)
        state["prompts"] = stream[:case["batch"] * case["prompt"]].reshape(case["batch"], case["prompt"])
        state["uniforms"] = rng.random((case["new"], case["batch"]))
        return state
    _random_weights(engine, case, gen)
    if train:
        if case["host_batches"]:  # one update's batches; a window's targets are its tokens moved by one
            start = rng.integers(0, stream.size - seq - 1, size=(case["accum"], case["batch"]))
            at = start[:, :, None] + np.arange(seq)
            state["batches"] = list(zip(stream[at], stream[at + 1]))
    else:
        state["windows"] = stream[rng.integers(0, stream.size - seq, size=case["windows"])[:, None] + np.arange(seq)]
    torch.cuda.synchronize()
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------
class Updated(dict):
    """Losses, weights and Adam's first moments after an update, by kind of tensor, all layers of a kind in one array.

    A training program leaves the last two where they are, in the engine's buffers on the GPU; here, too, a value is
    read from there when it is looked up.  (After the first update the moments are the clipped gradient times 0.1;
    Adam's second moments hold the same gradient squared.)"""

    KINDS = ("EMBED", "WQ", "WK", "WV", "WO", "W1", "W2", "W3", "RMS_ATT", "RMS_FFN", "RMS_FINAL", "VE_EMBED", "VE_GATE",
             "RESID_LAMBDAS", "X0_LAMBDAS", "SMEAR_GATE", "SMEAR_LAMBDA", "BACKOUT_LAMBDA")
    ONE = ("EMBED", "RMS_FINAL", "RESID_LAMBDAS", "X0_LAMBDAS", "SMEAR_GATE", "SMEAR_LAMBDA", "BACKOUT_LAMBDA")

    def __init__(self, engine, layers, losses):
        super().__init__(loss=losses)
        self.engine, self.layers = engine, layers
        for kind in self.KINDS:
            tid = getattr(ane, "T_" + kind)
            at = [n for n in range(1 if kind in self.ONE else layers) if engine.tensor_size(tid, n) > 0]
            if at:
                self["weight " + kind] = (tid, at, ane.engine.W)
                self["moment " + kind] = (tid, at, ane.engine.M)

    def __getitem__(self, key):
        value = super().__getitem__(key)
        if key == "loss":
            return value
        tid, at, which = value
        return np.concatenate([self.engine.export_tensor(tid, n, which) for n in at])


def run(state):
    case, engine = state["case"], state["engine"]
    if case["do"] == "train":
        if case["host_batches"]:
            losses = [engine.step_tokens(inp, tgt).loss for inp, tgt in state["batches"]]
        else:
            losses = [engine.step().loss for _ in range(case["accum"])]
        if "updated" not in state:
            state["updated"] = Updated(engine, case["layers"], [])
        state["updated"]["loss"] = losses
        return state["updated"]
    if case["do"] == "loss":
        return engine.eval_loss(state["windows"])
    if case["do"] == "logits":
        return engine.eval_logits(state["windows"])
    if case["temperature"] > 0:
        return engine.decode_sample(state["prompts"], case["new"], case["temperature"], state["uniforms"])
    return engine.decode_greedy(state["prompts"], case["new"])


# ---- the least work of one pass -------------------------------------------------------------------------------------
def _matrix_parameters(case):
    """Parameters that take part in a product, and all of them."""
    dim, hidden, layers, vocab = case["dim"], case["hidden"], case["layers"], case["vocab"]
    kv_dim = case["kv_heads"] * (dim // case["heads"])
    llama = case["arch"] == "llama"
    matrices = layers * (2 * dim * dim + 2 * dim * kv_dim + (3 if llama else 2) * dim * hidden) + vocab * dim
    if llama:
        return matrices, matrices + (2 * layers + 1) * dim
    tables = sum(1 for n in range(layers) if n % 2 == (layers - 1) % 2)  # value embeddings sit on every other layer
    return matrices + dim * dim, matrices + dim * dim + tables * vocab * dim


def work(case):
    matrices, everything = _matrix_parameters(case)
    dim, layers, seq, vocab = case["dim"], case["layers"], case["seq"], case["vocab"]
    width = 2 if case["dtype"] == "bf16" else 4
    if case["do"] == "train":  # weights and both moments in fp32, read and written; causal attention counted at half
        tokens = case["accum"] * case["batch"] * seq
        return {"bytes": 24 * everything + 4 * tokens, "flops": tokens * (6 * matrices + 3.5 * 2 * layers * seq * dim)}
    if case["do"] in ("loss", "logits"):
        tokens = case["windows"] * seq
        out = 4 * vocab * tokens if case["do"] == "logits" else 8
        return {"bytes": width * matrices + 2 * tokens + out, "flops": tokens * (2 * matrices + 2 * layers * seq * dim)}
    # every generated token needs all weights (once for the batch) and the keys and values so far (per sequence)
    batch, prompt, new = case["batch"], case["prompt"], case["new"]
    kv_dim = case["kv_heads"] * (dim // case["heads"])
    positions = (new - 1) * prompt + (new - 1) * new // 2
    kv_bytes = 2 * width * layers * kv_dim * batch * (positions + prompt)
    flops = batch * (prompt * (2 * (matrices - vocab * dim) + 2 * layers * prompt * dim) + new * 2 * vocab * dim
                     + (new - 1) * 2 * (matrices - vocab * dim) + 4 * layers * dim * positions)
    return {"bytes": width * matrices * new + kv_bytes, "flops": flops}


def tolerance(case):
    if case["do"] == "decode":
        return {"rel": 0.0, "differ": 0.01}  # the next token is clear of the others; a tie or a draw on an edge may fall otherwise
    if case["do"] == "loss":  # a sum over thousands of positions, each off by bf16 rounding of its own sign
        return {"rel": 1e-3}
    if case["do"] == "logits":
        return {"rel": 1e-2}
    if case["dtype"] == "bf16":
        # A weight gradient is a product of two chains of bf16 roundings, each about 1e-2 long in twelve layers; its
        # small elements beside large ones in the same row are off by a share of the row's, not of their own.
        return {"rel": 0.025, "max": 0.99}
    if case["dtype"] == "bf16x3":  # operands of 16 bits, and the softmax of unscaled scores multiplies what they drop
        return {"rel": 1e-3, "max": 0.3}
    # fp32 sums; an element whose gradient is within their rounding of zero is moved by the learning rate either way
    return {"rel": 1e-4, "max": 0.1}
