"""KV-cache greedy decoding (llama-style architecture, GQA) against full-recompute forwards.

fp32: every generated token equals the argmax of the oracle's full forward over the growing sequence
(argmax is an index path: bit-exact).  bf16: the cached path equals the engine's own full-recompute
EvalLogits argmax wherever the top-2 margin is clear."""
import numpy as np
import pytest

import ane
from oracle import oracle as O
from parity_utils import make_pair

pytestmark = pytest.mark.gpu


def test_decode_fp32_matches_oracle_full_recompute():
    cfg = dict(dim=64, hidden=96, heads=4, kv_heads=2, layers=3, vocab=256, seq=48)
    m, e = make_pair(ane, cfg, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_F32, batch=3, std=0.3, debug_taps=False)
    prompts = O.zipf_tokens(3 * 20, cfg["vocab"], 8).reshape(3, 20)
    n_new = 12
    got = e.decode_greedy(prompts, n_new)
    for b in range(3):
        seq = list(prompts[b])
        for step in range(n_new):
            padded = np.zeros(cfg["seq"], dtype=np.uint16)
            padded[:len(seq)] = seq                      # causal: later positions do not matter
            logits = m.eval_logits(padded)               # [vocab, seq]
            want = int(O.lib().orc_argmax(np.ascontiguousarray(logits[:, len(seq) - 1]).ctypes.data_as(
                __import__("ctypes").POINTER(__import__("ctypes").c_float)), cfg["vocab"]))
            assert int(got[b, step]) == want, (b, step)
            seq.append(want)
    e.close()


def test_decode_bf16_matches_own_full_forward():
    cfg = dict(dim=256, hidden=512, heads=4, kv_heads=2, layers=3, vocab=2048, seq=128)
    _, e = make_pair(ane, cfg, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_BF16, batch=4, std=0.08, debug_taps=False)
    prompts = O.zipf_tokens(4 * 64, cfg["vocab"], 9).reshape(4, 64)
    n_new = 24
    got = e.decode_greedy(prompts, n_new)
    agree = total = 0
    for b in range(4):
        full = np.zeros(cfg["seq"], dtype=np.uint16)
        full[:64] = prompts[b]
        full[64:64 + n_new] = got[b]
        logits = e.eval_logits(full)[0]                  # teacher-forced on the generated tokens
        for step in range(n_new):
            col = logits[:, 63 + step]
            top2 = np.sort(col)[-2:]
            if top2[1] - top2[0] > 0.05:                 # clear margin: bf16 noise cannot flip it
                total += 1
                agree += int(col.argmax() == got[b, step])
    assert total > 0 and agree == total
    with pytest.raises(ane.EngineError):
        e.decode_greedy(prompts, 100)                    # prompt_len + n_new > seq
    e.close()


def test_decode_bf16_gqa_full_size_batch_32_prompt_512():
    """The decode configuration at full size: 110M GQA model (12 query / 4 KV heads, 12 layers, vocab 32000, KV cache
    of 1024 positions), 32 sequences, 512-token prompts (prefill through the tcgen05 attention kernels, four 128-row
    tiles), then KV-cached greedy steps.  Checked against the engine's own full-recompute forward on four of the
    sequences: wherever the top-2 margin is clear the cached path picks the same token."""
    cfg = dict(dim=768, hidden=2048, heads=12, kv_heads=4, layers=12, vocab=32000, seq=1024)
    _, e = make_pair(ane, cfg, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_BF16, batch=32, std=0.05, debug_taps=False)
    prompts = O.zipf_tokens(32 * 512, cfg["vocab"], 12).reshape(32, 512)
    n_new = 24
    got = e.decode_greedy(prompts, n_new)
    assert got.shape == (32, n_new) and got.max() < cfg["vocab"]
    agree = total = 0
    for b in (0, 7, 19, 31):
        full = np.zeros(cfg["seq"], dtype=np.uint16)
        full[:512] = prompts[b]
        full[512:512 + n_new] = got[b]
        logits = e.eval_logits(full)[0]                  # [vocab, seq], teacher-forced on the generated tokens
        for step in range(n_new):
            col = logits[:, 511 + step]
            top2 = np.sort(col)[-2:]
            if top2[1] - top2[0] > 0.05:
                total += 1
                agree += int(col.argmax() == got[b, step])
    print(f"decode agreement {agree}/{total} on clear margins")
    assert total >= 8 and agree == total
    e.close()


def test_decode_rejected_for_reference_arch():
    cfg = dict(dim=64, hidden=96, heads=4, layers=2, vocab=256, seq=32)
    _, e = make_pair(ane, cfg, arch=O.ARCH_N, quirks=1, dtype=ane.DTYPE_F32, batch=1, debug_taps=False)
    with pytest.raises(ane.EngineError):
        e.decode_greedy(np.zeros((1, 8), np.uint16), 4)
    e.close()


def _upload(lib, a):
    p = lib.ane_dev_malloc(a.nbytes)
    assert lib.ane_dev_h2d(p, a.ctypes.data, a.nbytes) == 0
    return p


def test_sampler_rows_match_oracle_serial_walk():
    """sampleFromLogits (ane/train_full.go:318-342) is an index path: the device's chunked double sums must
    land on the oracle's index for the same uniform draw (a different index needs the target within double
    rounding of a prefix boundary, which seeded draws do not hit)."""
    import ctypes
    from ane import _ffi
    lib = _ffi.lib
    rng = np.random.default_rng(11)
    rows, vocab = 16, 32000
    logits = (4.0 * rng.standard_normal((rows, vocab))).astype(np.float32)
    logits[3, :] = 0.25                       # flat row: every index equally likely
    logits[4, 100] = 60.0                     # one dominant logit
    d_logits = _upload(lib, logits)
    d_out = lib.ane_dev_malloc(4 * rows)
    fp = ctypes.POINTER(ctypes.c_float)
    for temp in (0.0, 0.7, 1.0, 1.8):
        for trial in range(3):
            u = rng.random(rows)
            if trial == 0:
                u[:3] = (0.0, 1.0 - 2.0 ** -53, 0.5)
            d_u = _upload(lib, u)
            assert lib.ane_op_sample_rows(d_logits, d_u, temp, d_out, rows, vocab) == 0, lib.ane_ops_last_error()
            got = np.zeros(rows, dtype=np.int32)
            assert lib.ane_dev_d2h(got.ctypes.data, d_out, got.nbytes) == 0
            for r in range(rows):
                want = O.lib().orc_sample(logits[r].ctypes.data_as(fp), vocab, temp, float(u[r]))
                assert int(got[r]) == want, (temp, trial, r)
            lib.ane_dev_free(d_u)
    lib.ane_dev_free(d_logits)
    lib.ane_dev_free(d_out)


def test_decode_sample_fp32_matches_oracle_full_recompute():
    import ctypes
    cfg = dict(dim=64, hidden=96, heads=4, kv_heads=2, layers=3, vocab=256, seq=48)
    m, e = make_pair(ane, cfg, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_F32, batch=3, std=0.3, debug_taps=False)
    prompts = O.zipf_tokens(3 * 20, cfg["vocab"], 8).reshape(3, 20)
    n_new, temp = 10, 0.9
    u = np.random.default_rng(21).random((n_new, 3))
    got = e.decode_sample(prompts, n_new, temp, u)
    fp = ctypes.POINTER(ctypes.c_float)
    for b in range(3):
        seq = list(prompts[b])
        for step in range(n_new):
            padded = np.zeros(cfg["seq"], dtype=np.uint16)
            padded[:len(seq)] = seq
            col = np.ascontiguousarray(m.eval_logits(padded)[:, len(seq) - 1])
            want = O.lib().orc_sample(col.ctypes.data_as(fp), cfg["vocab"], temp, float(u[step, b]))
            if int(got[b, step]) != want:
                # fp32 GEMM summation order moves the logits by ~1e-6: accept a neighbour only when the draw sits
                # on that boundary
                w = np.exp((col.astype(np.float64) - col.max()) / temp)
                cum = np.cumsum(w) / w.sum()
                assert abs(cum[min(want, int(got[b, step]))] - u[step, b]) < 1e-5, (b, step)
            seq.append(int(got[b, step]))
    assert (e.decode_sample(prompts, n_new, 0.0, u) == e.decode_greedy(prompts, n_new)).all()
    with pytest.raises(ane.EngineError):
        e.decode_sample(prompts, n_new, temp, u[:, :2])
    e.close()


@pytest.mark.parametrize("batch,dim,heads,kv,hidden,vocab,prompt,temp", [
    (1, 128, 2, 1, 256, 512, 5, 0.0),       # one sequence; and the largest of its kernel
    (8, 192, 4, 2, 256, 504, 40, 0.9),      # head size 48
    (9, 128, 2, 1, 256, 512, 33, 0.0),      # smallest batch of the kernel for more, sixteen-row tile half empty
    (16, 64, 1, 1, 64, 96, 130, 0.9),       # fewer units of work than clusters; more keys than one round of the warps
    (17, 288, 6, 6, 768, 1000, 17, 0.0),    # contraction of 9 chunks: the last CTA of a cluster has none
    (32, 200, 5, 5, 544, 512, 12, 0.9),     # head size 40, contraction not a multiple of 32
    (32, 256, 2, 1, 2304, 512, 70, 0.0),    # head size 128; W2 in two boxes a row
    (33, 1280, 20, 4, 1024, 512, 20, 0.0),  # a second pass with one sequence; a norm read in two pieces
    (2, 512, 8, 8, 1376, 256, 5, 0.0),      # fewer units of the vocabulary than CTAs: some own none
    (12, 512, 8, 8, 1376, 96, 5, 0.0),      # and fewer than clusters
])
def test_decode_bf16_kernels_match_own_full_forward(batch, dim, heads, kv, hidden, vocab, prompt, temp):
    """Tokens of the persistent kernels against the engine's full forward over prompt + generated tokens.

    Two chains of bf16 roundings of the same values differ in a logit by about 2^-8 sqrt(dim) std (an element of the
    normalised row is 1, of the classifier std) times the root of some 8 roundings per layer that feed it; `tol` is six of
    that.  Greedy: the token's logit is within tol of the best (a wrong value somewhere costs units).  Sampled: the draw
    lies in the token's interval of the distribution, whose edges move by at most a factor e^(2 tol / T)."""
    layers, new, std = 3, 12, 0.08
    seq = (prompt + new + 63) // 64 * 64
    cfg = dict(dim=dim, hidden=hidden, heads=heads, kv_heads=kv, layers=layers, vocab=vocab, seq=seq)
    _, e = make_pair(ane, cfg, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_BF16, batch=batch, std=std, debug_taps=False)
    prompts = O.zipf_tokens(batch * prompt, vocab, 3).reshape(batch, prompt)
    u = np.random.default_rng(5).random((new, batch))
    got = e.decode_sample(prompts, new, temp, u) if temp > 0 else e.decode_greedy(prompts, new)
    full = np.zeros((batch, seq), np.uint16)
    full[:, :prompt], full[:, prompt:prompt + new] = prompts, got
    tol = 6 * 2.0 ** -8 * np.sqrt(dim) * std * np.sqrt(8 * layers)
    for b in range(batch):
        logits = e.eval_logits(full[b])[0][:, prompt - 1:prompt + new - 1].astype(np.float64)
        for step in range(new):
            col, tok = logits[:, step], int(got[b, step])
            if temp == 0:
                assert col.max() - col[tok] <= tol, (b, step)
            else:
                p = np.exp((col - col.max()) / temp)
                at, total = np.cumsum(p), p.sum()
                slack = np.expm1(2 * tol / temp)
                assert (at[tok] - p[tok]) / total - slack <= u[step, b] <= at[tok] / total + slack, (b, step)


@pytest.mark.parametrize("batch,dim,heads,kv,hidden,vocab,new,temp", [
    (1, 288, 6, 2, 768, 32000, 24, 1.0),     # kernel for up to eight sequences, fewer CTAs than SMs
    (8, 288, 6, 3, 768, 4096, 24, 0.7),
    (4, 768, 12, 4, 2048, 32000, 24, 1.0),   # on all SMs
    (9, 288, 6, 6, 768, 32000, 24, 1.0),     # cluster kernel
    (20, 288, 6, 2, 768, 4096, 24, 0.7),
    (32, 768, 12, 4, 2048, 32000, 24, 1.0),
    (2, 512, 8, 8, 1376, 256, 24, 1.0),      # fewer units of the vocabulary than CTAs: some own none
    (2, 512, 8, 8, 1376, 256, 2, 0.7),
    (12, 512, 8, 8, 1376, 96, 24, 0.7),
])
def test_sampled_tokens_are_the_serial_walks(batch, dim, heads, kv, hidden, vocab, new, temp):
    """The sampler of the persistent kernels, index by index.  All weights but the embedding are zero, so the stream stays the
    token's embedding; its elements are +-1/64, normalised they are +-c for one bf16 number c, and a logit is c / 64 times a whole
    number: exact in fp32 in any order of addition.  The token must be the one of the serial walk in double over those logits
    (ane/train_full.go:318-342).  Draws: 0, the largest below 1, 1e-9 to either side of the edges of CTA ranges (sums in another
    order move an edge by 1e-13), and random ones."""
    a, prompt = 1.0 / 64, 3
    rng = np.random.default_rng(vocab + batch)
    signs = rng.integers(0, 2, (vocab, dim)).astype(np.float32) * 2 - 1
    x = np.float32(a) * (np.float32(1) / np.sqrt(np.float32(a * a) + np.float32(1e-5)))
    c = float(np.float32(np.round(float(x) * 256) / 256))  # 8 bits in [1/2, 1)
    assert abs(abs(float(x) - c) - 1 / 512) > 1e-4         # clear of a rounding edge
    e = ane.open(ane.Options(dim=dim, hidden=hidden, n_layers=2, n_heads=heads, n_kv_heads=kv, vocab=vocab, seq=64, batch=batch,
                             arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16))
    e.import_tensor(ane.T_EMBED, 0, signs * np.float32(a))
    prompts = rng.integers(0, vocab, (batch, prompt)).astype(np.uint16)
    units = vocab // 8
    edges = sorted({8 * (units * i // n) for n in (60, 132, 136, 140, 144, 148) for i in range(1, n)} - {0})
    u, want = np.zeros((new, batch)), np.zeros((batch, new), np.uint16)
    last = prompts[:, -1].astype(int)
    inv_temp = float(np.float32(1) / np.float32(temp))
    for step in range(new):
        logits = (signs @ signs[last].T).astype(np.float64) * (c * a)  # whole numbers up to dim: exact
        cdf = np.cumsum(np.exp((logits - logits.max(0)) * inv_temp), 0)
        for b in range(batch):
            kind = (step + b) % 6
            at = cdf[edges[rng.integers(len(edges))] - 1, b] / cdf[-1, b]
            u[step, b] = (0.0, 1 - 2.0 ** -53, at - 1e-9, at + 1e-9, rng.random(), rng.random())[kind]
            want[b, step] = min(int(np.searchsorted(cdf[:, b], u[step, b] * cdf[-1, b])), vocab - 1)
        last = want[:, step].astype(int)
    got = e.decode_sample(prompts, new, temp, u)
    e.close()
    np.testing.assert_array_equal(got, want)


def test_decode_after_its_buffers_could_not_be_allocated():
    """The first decode allocates the caches and its scratch.  With memory left for the two caches (128 MiB each) but not for
    all of the rest (8 MiB of draws) it reports an error and keeps nothing; when there is memory again it decodes."""
    from ane import _ffi
    lib = _ffi.lib
    opts = ane.Options(dim=64, hidden=64, n_layers=1, n_heads=1, n_kv_heads=1, vocab=96, seq=512, batch=2048, arch=ane.ARCH_LLAMA,
                       quirks=0, compute_dtype=ane.DTYPE_BF16)
    weights = np.random.default_rng(3).standard_normal((96, 64)).astype(np.float32)
    prompts = O.zipf_tokens(2 * 8, 96, 3).reshape(2, 8)
    e = ane.open(opts)
    e.import_tensor(ane.T_EMBED, 0, weights)
    room = lib.ane_dev_malloc(260 << 20)
    held, size = [], 1 << 34
    while size >= 1 << 20:
        p = lib.ane_dev_malloc(size)
        if p:
            held.append(p)
        else:
            size >>= 1
    lib.ane_dev_free(room)
    try:
        with pytest.raises(ane.EngineError, match="cudaMalloc"):
            e.decode_greedy(prompts, 4)
        with pytest.raises(ane.EngineError, match="cudaMalloc"):
            e.decode_greedy(prompts, 4)
    finally:
        for p in held:
            lib.ane_dev_free(p)
    got = e.decode_greedy(prompts, 4)
    e.close()
    e = ane.open(opts)
    e.import_tensor(ane.T_EMBED, 0, weights)
    np.testing.assert_array_equal(got, e.decode_greedy(prompts, 4))
    e.close()


def _decode_in_a_child(env):
    """Tokens of 2 greedy and 36 sampled sequences, from a process with `env`."""
    import json
    import os
    import subprocess
    import sys
    code = """
import json, sys
import numpy as np
import ane
rng = np.random.default_rng(4)
out = []
for batch, temp in ((2, 0.0), (36, 0.9)):
    e = ane.open(ane.Options(dim=128, hidden=256, n_layers=2, n_heads=2, n_kv_heads=1, vocab=512, seq=64, batch=batch, arch=ane.ARCH_LLAMA,
                             quirks=0, compute_dtype=ane.DTYPE_BF16))
    e.import_tensor(ane.T_EMBED, 0, (rng.integers(0, 2, (512, 128)) * 2 - 1).astype(np.float32) / 64)
    prompts = rng.integers(0, 512, (batch, 5)).astype(np.uint16)
    before = e.launch_count()
    tokens = e.decode_sample(prompts, 9, temp, rng.random((9, batch)))
    out.append([tokens.tolist(), e.launch_count() - before])
    e.close()
print(json.dumps(out))
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "autoresearch-go-ane_b200"), **env)
    done = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    return json.loads(done.stdout.strip().splitlines()[-1])


def test_decode_where_the_persistent_kernel_does_not_fit():
    """On two SMs (ANE_B200_GEMM_SMS) there is no cluster of four CTAs to launch, a launch that the host refuses; decoding goes
    one step after the other then.  Zero weights but the embedding: logits are exact, so the tokens are the same."""
    whole, two = _decode_in_a_child({}), _decode_in_a_child({"ANE_B200_GEMM_SMS": "2"})
    for (tokens, launches), (same, more) in zip(whole, two):
        assert same == tokens
        assert more > 2 * launches


@pytest.mark.parametrize("batch", [2, 9])
def test_norm_of_a_row_whose_squares_overflow(batch):
    """A row with a sum of squares beyond fp32 is normalised to zeros (1 / sqrt(inf)), in the persistent kernels as in prefill and
    step by step.  All weights but the embedding are zero, so the stream is the token's embedding: after BIG all logits are 0
    (index 0), after 0 the largest is NEXT's, after NEXT it is BIG's."""
    dim, vocab, prompt, new = 128, 96, 3, 9
    big, nxt = 5, 7
    embed = np.full((vocab, dim), 1.0 / 64, np.float32)
    embed[:, 0] = 0
    embed[0], embed[nxt], embed[big] = 0, 0, 0
    embed[0, 0], embed[0, 1] = -1, 8
    embed[nxt, 0], embed[nxt, 1] = 1, 16
    embed[big, 0] = 1e20
    e = ane.open(ane.Options(dim=dim, hidden=256, n_layers=2, n_heads=2, n_kv_heads=2, vocab=vocab, seq=64, batch=batch,
                             arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16))
    e.import_tensor(ane.T_EMBED, 0, embed)
    got = e.decode_greedy(np.full((batch, prompt), nxt, np.uint16), new)
    e.close()
    np.testing.assert_array_equal(got, np.tile(np.array([big, 0, nxt], np.uint16), (batch, 3)))
