"""GPU checks of the callers around the step: the training driver and evaluation harness on a real engine,
Open with a model path (llama2.c model file, else a checkpoint: ane/engine.go:250-257), and what
LoadCheckpoint does beyond copying tensors (sampler reseed, wall clock: ane/engine.go:559-560)."""
import struct

import numpy as np
import pytest

import ane
from ane import checkpoint as C
from ane import harness as H
from oracle import oracle as O
from parity_utils import make_pair, rel_l2

pytestmark = pytest.mark.gpu

CFG = dict(dim=64, hidden=96, heads=4, layers=3, vocab=256, seq=32)


def _options(cfg, **kw):
    return ane.Options(dim=cfg["dim"], hidden=cfg["hidden"], n_layers=cfg["layers"], n_heads=cfg["heads"],
                       n_kv_heads=cfg.get("kv_heads", cfg["heads"]), vocab=cfg["vocab"], seq=cfg["seq"], **kw)


@pytest.mark.parametrize("arch,quirks", [(O.ARCH_N, 1), (O.ARCH_L, 0)])
def test_training_driver_and_evaluation_harness_on_an_engine(arch, quirks):
    """harness.train for six counted steps (after its three warm-up steps) with the schedule's learning rates
    set before every step, then eval_loss / val_bpb over the validation windows against the oracle's
    window loss on the engine's own trained weights."""
    toks = O.zipf_tokens(4096, CFG["vocab"], 17)
    hyper = dict(lr=1e-3, adam_beta1=0.9, adam_beta2=0.95, weight_decay=0.1, grad_clip=1.0, accum_steps=2)
    m, e = make_pair(ane, CFG, arch=arch, quirks=quirks, dtype=ane.DTYPE_F32, batch=2, hyper=hyper, tokens=toks,
                     debug_taps=False, std=0.1)
    log = H.train(e, max_steps=6, peak_lr=1e-3)
    assert log.steps == 6 and log.tokens == 6 * 2 * CFG["seq"] and len(log.losses) == 6
    assert all(np.isfinite(l) for l in log.losses)
    st = e.state()
    assert st.cum_steps == 6 + H.WARMUP_STEPS and st.pending_steps == 0          # train() ends with a flush
    assert st.adam_t == 5                                                        # 9 micro-steps of 2: 4 updates + the final flush
    assert log.lrs[0] == pytest.approx(1e-6) and log.lrs[1] == pytest.approx(H.lr_schedule(1 / 6, 1e-3))
    assert e.lr() == pytest.approx(log.lrs[-1])
    # evaluation: the harness's windows over the last 600 tokens, fused device loss against the oracle on the
    # same (trained) weights
    for tid, layer, a in m.tensors(O.W):
        a[:] = e.export_tensor(tid, layer).reshape(a.shape)
    got = H.eval_loss(e, toks, eval_tokens=600)
    windows = H.eval_windows(toks, 600, CFG["seq"])
    assert len(windows) == 19                                                    # starts 0, 31, ..., 558
    tot, n = 0.0, 0
    for w in windows:
        s, k = m.eval_loss_window(np.ascontiguousarray(w))
        tot, n = tot + s, n + k
    assert got == pytest.approx(tot / n, abs=1e-4)
    assert H.val_bpb(got) == pytest.approx(got / np.log(2.0) / 3.7)
    # the reference's own (mis-indexed) walk over downloaded logits, reproduced from the oracle's logits
    ref_walk = H.eval_loss(e, toks, eval_tokens=600, reference_indexing=True)

    class OracleLogits:
        seq, vocab, opts = CFG["seq"], CFG["vocab"], e.opts

        def eval_logits(self, w, layout=0):
            return m.eval_logits(np.ascontiguousarray(w))[None]

    assert ref_walk == pytest.approx(H.eval_loss(OracleLogits(), toks, eval_tokens=600, reference_indexing=True), abs=1e-4)
    e.close()


def test_benchmarks_with_the_reference_metric_names_on_an_engine():
    """The three benchmarks of bench_test.go:75-158 through the harness twins on a real engine: metric names,
    consistency of tok/s with the step's own duration, val_bpb from val_loss."""
    toks = O.zipf_tokens(4096, CFG["vocab"], 19)
    hyper = dict(lr=1e-3, accum_steps=2)
    m, e = make_pair(ane, CFG, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_F32, batch=2, hyper=hyper, tokens=toks,
                     debug_taps=False, std=0.1)
    b = H.benchmark_step(e, n=4)
    assert set(b) >= {"loss", "tok/s", "tok/s_processed", "step_ms", "ane_ms", "adam_ms", "ns/op"}
    assert np.isfinite(b["loss"]) and b["step_ms"] > 0 and 0 < b["ane_ms"] <= b["step_ms"] + 1e-6
    assert b["tok/s"] == pytest.approx(CFG["seq"] * 2 / (b["step_ms"] * 1e-3))
    assert b["tok/s_processed"] == pytest.approx(2 * CFG["seq"] / (b["step_ms"] * 1e-3))
    assert e.state().cum_steps == 7
    lg = H.benchmark_eval_logits(e, toks, n=3, seq=CFG["seq"])
    assert lg["ns/op"] > 0 and lg["tok/s"] == pytest.approx(CFG["seq"] / (lg["ns/op"] * 1e-9))
    ev = H.benchmark_eval_loss(e, toks, eval_tokens=600)
    assert ev["val_loss"] == pytest.approx(H.eval_loss(e, toks, eval_tokens=600), abs=1e-6)
    assert ev["val_bpb"] == pytest.approx(ev["val_loss"] / np.log(2.0) / 3.7)
    e.close()


def test_eval_logits_into_page_locked_memory_matches_the_staged_copy():
    """ane.pinned_empty gives page-locked memory; EvalLogits copies into it straight from the device and must
    return what the staged path (pageable array) returns, in both layouts and for several windows."""
    toks = O.zipf_tokens(4096, CFG["vocab"], 23)
    m, e = make_pair(ane, CFG, arch=O.ARCH_L, quirks=0, dtype=ane.DTYPE_F32, batch=2, hyper=dict(lr=1e-3), tokens=toks,
                     debug_taps=False, std=0.1)
    windows = np.ascontiguousarray(toks[:3 * CFG["seq"]])
    for layout in (0, 1):
        want = e.eval_logits(windows, layout=layout)
        out = ane.pinned_empty(want.shape)
        out[...] = -1.0
        got = e.eval_logits(windows, layout=layout, out=out)
        assert got is out
        np.testing.assert_array_equal(got, want)
    del out, got
    e.close()


def test_load_checkpoint_reseeds_the_sampler_and_keeps_the_wall_clock(tmp_path):
    toks = O.zipf_tokens(8192, CFG["vocab"], 5)
    hyper = dict(lr=1e-3, accum_steps=1, seed=7)
    _, first = make_pair(ane, CFG, arch=O.ARCH_N, quirks=1, dtype=ane.DTYPE_F32, batch=2, hyper=hyper, tokens=toks,
                         debug_taps=False)
    for _ in range(3):
        first.step()
    wall = first.state().cum_wall_ms
    path = str(tmp_path / "r.ckpt")
    C.save_checkpoint(first, path, C.TrainMeta(step=3))
    first.close()
    _, second = make_pair(ane, CFG, arch=O.ARCH_N, quirks=1, dtype=ane.DTYPE_F32, batch=2, hyper=hyper, tokens=toks,
                          debug_taps=False)
    C.load_checkpoint(second, path)
    second.step()
    # ane/engine.go:559: the resumed stream is drand48Seed(seed + meta.Step), not a replay of the first run
    want = O.drand48_positions(7 + 3, toks.size, CFG["seq"], 2)
    assert second.state().token_pos == want[1] + CFG["seq"]
    replay = O.drand48_positions(7, toks.size, CFG["seq"], 2)
    assert want[1] != replay[1]
    assert second.state().cum_wall_ms >= wall                                     # ane/engine.go:560
    second.close()


def test_open_with_a_model_path_reads_a_model_file_or_a_checkpoint(tmp_path):
    cfg = dict(CFG)
    rng = np.random.default_rng(2)
    L, V, D, Hd, H_ = cfg["layers"], cfg["vocab"], cfg["dim"], cfg["hidden"], cfg["heads"]
    parts = dict(embed=(V * D,), rms_att=(L, D), wq=(L, D * D), wk=(L, D * D), wv=(L, D * D), wo=(L, D * D),
                 rms_ffn=(L, D), w1=(L, Hd * D), w2=(L, D * Hd), w3=(L, Hd * D), rms_final=(D,))
    data = {k: (0.05 * rng.standard_normal(s)).astype(np.float32) for k, s in parts.items()}
    model = str(tmp_path / "model.bin")
    with open(model, "wb") as f:
        f.write(struct.pack("<7i", D, Hd, L, H_, H_, V, cfg["seq"]))
        for k in parts:
            data[k].tofile(f)
    e = ane.open(_options(cfg, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_F32, batch=1, model_path=model))
    np.testing.assert_array_equal(e.export_tensor(ane.T_WK, 2), data["wk"][2])
    np.testing.assert_array_equal(e.export_tensor(ane.T_W3, 1), data["w3"][1])
    np.testing.assert_array_equal(e.export_tensor(ane.T_RMS_FINAL, 0), data["rms_final"])
    # the same weights saved as a checkpoint open again through the second branch of Open
    C.random_init(e, 4)
    ckpt = str(tmp_path / "init.ckpt")
    C.save_checkpoint(e, ckpt, C.TrainMeta(step=0, lr=3e-4))
    e2 = ane.open(_options(cfg, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_F32, batch=1, model_path=ckpt))
    for tid in (ane.T_EMBED, ane.T_WQ, ane.T_W2, ane.T_W3):
        np.testing.assert_array_equal(e2.export_tensor(tid, 1 if tid != ane.T_EMBED else 0),
                                      e.export_tensor(tid, 1 if tid != ane.T_EMBED else 0))
    window = O.zipf_tokens(cfg["seq"], V, 3)
    assert rel_l2(e2.eval_logits(window), e.eval_logits(window)) < 1e-6
    e.close()
    e2.close()
    with pytest.raises(ane.EngineError, match="load model"):
        ane.open(_options(cfg, arch=ane.ARCH_LLAMA, compute_dtype=ane.DTYPE_F32, batch=1,
                          model_path=str(tmp_path / "missing.bin")))
    junk = tmp_path / "junk.bin"
    junk.write_bytes(b"\x01" * 64)
    with pytest.raises(ane.EngineError, match="load model"):
        ane.open(_options(cfg, arch=ane.ARCH_LLAMA, compute_dtype=ane.DTYPE_F32, batch=1, model_path=str(junk)))


@pytest.mark.parametrize("dtype", [ane.DTYPE_BF16, ane.DTYPE_F32, ane.DTYPE_BF16X3])
def test_eval_loss_between_calls_that_need_more_scratch(dtype):
    """The evaluation loss is replayed from a graph from the second pass of a window count on; a step, EvalLogits and another
    window count in between (in split precision each has larger operands, whose scratch moves) must not change what it
    reads.  The same kernels on the same weights in the same order: equal to a fresh engine's first, eager pass."""
    toks = O.zipf_tokens(4096, CFG["vocab"], 29)
    seq = CFG["seq"]
    two, one = np.ascontiguousarray(toks[:2 * seq]), np.ascontiguousarray(toks[7 * seq:8 * seq])

    def fresh_loss(e, windows):
        _, f = make_pair(ane, CFG, arch=O.ARCH_N, quirks=0, dtype=dtype, batch=2, debug_taps=False)
        for tid, layer, a in m.tensors(O.W):
            f.import_tensor(tid, layer, e.export_tensor(tid, layer))
        loss = f.eval_loss(windows)
        f.close()
        return loss

    m, e = make_pair(ane, CFG, arch=O.ARCH_N, quirks=0, dtype=dtype, batch=2, hyper=dict(lr=1e-2, accum_steps=1), std=0.1,
                     tokens=toks, debug_taps=False)
    for _ in range(3):
        assert e.eval_loss(one) == fresh_loss(e, one)
    for between in (lambda: e.eval_loss(two), lambda: e.eval_logits(one, layout=1), lambda: e.eval_logits(one), e.step):
        between()
        for windows in (one, two):
            for _ in range(3):
                assert e.eval_loss(windows) == fresh_loss(e, windows)
    e.close()


def test_evaluation_loss_counts_a_tile_of_nan_logits():
    """256 embedding rows of NaN make a whole tile of the classifier's statistics NaN, without a maximum.  The softmax over the
    vocabulary is NaN then, and the loss of every position -log of the probability's floor of 1e-10 (ane/stories/cpu.go:212-292)."""
    e = ane.open(ane.Options(dim=64, hidden=64, n_layers=1, n_heads=1, n_kv_heads=1, vocab=1024, seq=32, batch=1, arch=ane.ARCH_LLAMA,
                             quirks=0, compute_dtype=ane.DTYPE_BF16))
    embed = (0.02 * np.random.default_rng(1).standard_normal((1024, 64))).astype(np.float32)
    window = np.arange(32, dtype=np.uint16)
    e.import_tensor(ane.T_EMBED, 0, embed)
    loss, n = e.eval_loss(window)
    assert n == 31 and loss / n == pytest.approx(np.log(1024), abs=0.1)
    for tile in range(1, 4):
        bad = embed.copy()
        bad[256 * tile:256 * (tile + 1)] = np.nan
        e.import_tensor(ane.T_EMBED, 0, bad)
        loss, n = e.eval_loss(window)
        assert n == 31 and loss / n == pytest.approx(-np.log(1e-10), abs=1e-3)
    e.close()


@pytest.mark.parametrize("vocab,seq", [(2048, 132), (4096, 96), (20008, 128)])
def test_eval_logits_by_several_threads(vocab, seq):
    """Windows of 1 to 10 MiB, copied by several threads in pieces and blocks that the size is no multiple of, into fresh memory and
    into the middle of an array whose other values must stay; against page-locked memory, which takes the download directly."""
    e = ane.open(ane.Options(dim=64, hidden=64, n_layers=1, n_heads=1, n_kv_heads=1, vocab=vocab, seq=seq, batch=2, arch=ane.ARCH_LLAMA,
                             quirks=0, compute_dtype=ane.DTYPE_BF16))
    e.import_tensor(ane.T_EMBED, 0, np.random.default_rng(7).standard_normal((vocab, 64)).astype(np.float32))
    for count in (1, 3):
        windows = O.zipf_tokens(count * seq, vocab, 11)
        want = e.eval_logits(windows, out=ane.pinned_empty((count, vocab, seq)))
        for _ in range(3):
            np.testing.assert_array_equal(e.eval_logits(windows), want)
            held = np.full(want.size + 12, -7.0, np.float32)
            e.eval_logits(windows, out=held[5:5 + want.size].reshape(want.shape))
            np.testing.assert_array_equal(held[5:-7], want.ravel())
            assert (held[:5] == -7).all() and (held[-7:] == -7).all()
    e.close()


@pytest.mark.parametrize("arch,dtype", [(ane.ARCH_LLAMA, ane.DTYPE_BF16), (ane.ARCH_REFERENCE, ane.DTYPE_BF16), (ane.ARCH_LLAMA, ane.DTYPE_BF16X3)])
def test_logits_of_a_window_do_not_depend_on_its_batch(arch, dtype):
    """Forward products on the tensor cores have one accumulator for the whole contraction, and the other kernels go row by row or
    head by head: the logits of a window are the same, bit for bit, alone and among others."""
    cfg = dict(dim=768, hidden=2048, heads=12, layers=2, vocab=512, seq=256)
    rng = np.random.default_rng(9)
    windows = O.zipf_tokens(24 * cfg["seq"], cfg["vocab"], 13)
    logits = []
    for batch in (1, 2, 24):
        e = ane.open(_options(cfg, batch=batch, arch=arch, quirks=0, compute_dtype=dtype))
        rng = np.random.default_rng(9)
        for tid in (ane.T_EMBED, ane.T_WQ, ane.T_WK, ane.T_WV, ane.T_WO, ane.T_W1, ane.T_W2) + ((ane.T_W3,) if arch == ane.ARCH_LLAMA else ()):
            for layer in range(1 if tid == ane.T_EMBED else cfg["layers"]):
                e.import_tensor(tid, layer, (0.05 * rng.standard_normal(e.tensor_size(tid, layer))).astype(np.float32))
        logits.append(e.eval_logits(windows)[:2])
        e.close()
    np.testing.assert_array_equal(logits[0], logits[1])
    np.testing.assert_array_equal(logits[0], logits[2])


F32_CFG = dict(dim=288, hidden=768, heads=6, layers=2, vocab=32000, seq=256)  # products that the tensor cores take in three parts


def _free_mib():
    import torch
    return torch.cuda.mem_get_info()[0] / 2**20


def _f32_engine(toks):
    e = ane.open(_options(F32_CFG, tokens=toks, batch=4, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_F32, accum_steps=1))
    C.random_init(e, 6)
    return e


def test_fp32_engines_take_their_memory_when_they_are_opened():
    """Updates, evaluation losses and logits of an fp32 engine allocate nothing (16 MiB for kernels that are loaded on their first
    launch), and it leaves nothing behind."""
    toks = O.zipf_tokens(1 << 14, F32_CFG["vocab"], 31)
    _f32_engine(toks).close()
    before = _free_mib()
    e = _f32_engine(toks)
    opened = _free_mib()
    for use in (e.step, lambda: e.eval_loss(toks[:1024]), lambda: e.eval_logits(toks[:256]), lambda: e.eval_logits(toks[:256], layout=1), e.step):
        use()
        assert abs(_free_mib() - opened) < 16
    e.close()
    assert abs(_free_mib() - before) < 16


def test_fp32_engine_without_memory_for_the_parts_of_its_operands():
    """An engine that fits without the parts opens where they do not fit, and stays on the FMA units without asking for memory again."""
    toks = O.zipf_tokens(1 << 14, F32_CFG["vocab"], 31)
    e = _f32_engine(toks)
    losses = [e.step().loss for _ in range(3)]
    held = _free_mib()
    e.close()
    free = _free_mib()
    parts = 2 * 6 * 1024 * 32000 / 2**20  # of d logits alone, on both streams
    filler = ane._ffi.lib.ane_dev_malloc(int((held + parts - 100) * 2**20))  # leaves the engine, and 100 MiB of these 375
    assert filler
    try:
        e = _f32_engine(toks)
        opened = _free_mib()
        assert opened > 40 and free - held > parts
        for want in losses:
            assert e.step().loss == pytest.approx(want, abs=1e-4)
            assert abs(_free_mib() - opened) < 16
        e.close()
    finally:
        ane._ffi.lib.ane_dev_free(filler)


def test_fp32_engine_gives_the_parts_of_its_operands_back_for_a_decode():
    """The caches of the first decode come after the parts: where only one of them fits, it is the caches.  Same tokens as with both, and
    the evaluation loss, a graph of the former scratch by then, within the rounding of the FMA units."""
    toks = O.zipf_tokens(1 << 14, F32_CFG["vocab"], 31)
    prompts = np.ascontiguousarray(toks[:64]).reshape(4, 16)
    cfg = dict(F32_CFG, seq=12288, vocab=512)  # caches of 216 MiB, logits of 24
    e = ane.open(_options(cfg, batch=4, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_F32))
    C.random_init(e, 6)
    tokens = e.decode_greedy(prompts % 512, 6)
    e.close()
    e = ane.open(_options(cfg, batch=4, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_F32))
    C.random_init(e, 6)
    window = np.ascontiguousarray(toks[:cfg["seq"]] % 512)
    losses = [e.eval_loss(window)[0] for _ in range(3)]
    caches = 2 * 4 * 4 * 2 * cfg["seq"] * cfg["dim"] / 2**20
    filler = ane._ffi.lib.ane_dev_malloc(int((_free_mib() - caches / 2) * 2**20))
    assert filler
    try:
        np.testing.assert_array_equal(e.decode_greedy(prompts % 512, 6), tokens)
        for _ in range(3):
            assert e.eval_loss(window)[0] == pytest.approx(losses[0], rel=1e-5)
        e.close()
    finally:
        ane._ffi.lib.ane_dev_free(filler)


@pytest.mark.parametrize("first", ["logits", "decode"])
def test_split_precision_engine_gives_its_halves_back(first):
    """What fits only without the kept halves of the operands gets their place: a larger scratch for the classifier product of EvalLogits,
    the caches of the first decode.  Whoever cuts them, the halves are the same: equal losses (a graph of the former halves by then),
    logits and tokens, and gradients but for the order of their atomic sums."""
    toks = O.zipf_tokens(1 << 14, F32_CFG["vocab"], 31)
    cfg = dict(F32_CFG, seq=1024)
    windows, prompts = toks[:3 * cfg["seq"]].reshape(3, -1), np.ascontiguousarray(toks[:64]).reshape(4, 16)
    results = []
    for left in (None, 32):  # MiB: the scratch takes 51 (and frees 12 first), the caches 151, the halves 500
        e = ane.open(_options(cfg, tokens=toks, batch=16, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16X3, accum_steps=1000, ce_chunk_rows=256))
        C.random_init(e, 6)
        out = [e.step().loss] + [e.eval_loss(windows)[0] for _ in range(3)]
        filler = ane._ffi.lib.ane_dev_malloc(int((_free_mib() - left) * 2**20)) if left else None
        assert filler or not left
        try:
            use = {"logits": lambda: e.eval_logits(windows[0]), "decode": lambda: e.decode_greedy(prompts, 5)}
            for name in sorted(use, key=lambda name: name != first):
                out.append(use[name]())
                assert not left or _free_mib() > 250
            out += [e.eval_loss(windows)[0] for _ in range(3)] + [e.step().loss]
            grads = [e.export_tensor(t, 0, O.G) for t in (ane.T_EMBED, ane.T_WQ, ane.T_W2)]
            e.close()
        finally:
            if filler:
                ane._ffi.lib.ane_dev_free(filler)
        results.append((out, grads))
    for a, b in zip(results[0][0], results[1][0]):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(results[0][1], results[1][1]):
        assert rel_l2(b, a) < 2e-6


@pytest.mark.parametrize("busy", [False, True])
def test_split_precision_engine_gives_its_halves_back_to_another_engine(busy):
    """An engine that fits only without the halves that another one holds opens, as soon as the other one is in no call (busy: a thread
    steps it all the while), and the other one goes on with the same losses."""
    import threading
    toks = O.zipf_tokens(1 << 14, F32_CFG["vocab"], 31)
    cfg = dict(F32_CFG, seq=1024)

    def holder():
        e = ane.open(_options(cfg, tokens=toks, batch=16, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16X3, accum_steps=1000, ce_chunk_rows=256))
        C.random_init(e, 6)
        return e

    def other():
        e = ane.open(_options(F32_CFG, tokens=toks, batch=4, arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16))
        C.random_init(e, 7)
        return e

    e = holder()
    free = _free_mib()
    second = other()
    takes = free - _free_mib()
    want = [e.step().loss for _ in range(12)], second.step().loss
    second.close()
    e.close()
    assert 100 < takes < 900  # (the halves are 500)
    e = holder()
    filler = ane._ffi.lib.ane_dev_malloc(int((_free_mib() - takes / 2) * 2**20))
    assert filler
    losses = []
    try:
        turns = threading.Thread(target=lambda: losses.extend(e.step().loss for _ in range(12)))
        if busy:
            turns.start()
        second = None
        while second is None:
            idle = not turns.is_alive()
            try:
                second = other()
            except ane.EngineError:
                assert not idle
        if not busy:
            turns.start()
        turns.join()
        assert losses == want[0] and second.step().loss == want[1]
        second.close()
        e.close()
    finally:
        ane._ffi.lib.ane_dev_free(filler)
