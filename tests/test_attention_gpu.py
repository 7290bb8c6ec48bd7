"""Attention kernels at the edges of their tiles, against the oracle: the fp32 kernels (32 resident rows, streamed tiles of
64, head sizes padded to 32 / 48 / 64 / 96 / 128) and the mma.sync kernels (head sizes 32, 48 and 64; 64- or 128-row blocks)."""
import numpy as np
import pytest

import ane
from oracle import oracle as O
from parity_utils import compare_grads, make_pair, oracle_batch_accumulate
from test_parity_gpu import BWD_TAPS, F32_TOL, FWD_TAPS, batch_tokens, tap_errors

pytestmark = pytest.mark.gpu


def _step(dtype, arch, quirks, hd, heads, kv, seq, batch, std):
    cfg = dict(dim=hd * heads, hidden=64, heads=heads, kv_heads=kv, layers=2, vocab=96, seq=seq)
    m, e = make_pair(ane, cfg, arch=arch, quirks=quirks, dtype=dtype, batch=batch, std=std,
                     hyper=dict(accum_steps=1000, grad_clip=1.0))
    inp, tgt = batch_tokens(cfg, batch, 7, invalid=False)
    r = e.step_tokens(inp, tgt)
    assert r.device_status == 0
    return cfg, m, e, inp, tgt


@pytest.mark.parametrize("arch,hd,heads,kv,seq", [
    (O.ARCH_L, 8, 2, 1, 31), (O.ARCH_L, 32, 2, 2, 33), (O.ARCH_L, 48, 2, 1, 64), (O.ARCH_L, 64, 1, 1, 65), (O.ARCH_L, 72, 2, 1, 97),
    (O.ARCH_L, 128, 2, 1, 130), (O.ARCH_N, 48, 2, 2, 129), (O.ARCH_N, 104, 1, 1, 63)])
def test_fp32_tiles(arch, hd, heads, kv, seq):
    cfg, m, e, inp, tgt = _step(ane.DTYPE_F32, arch, int(arch == O.ARCH_N), hd, heads, kv, seq, 2, 0.1)
    oracle_batch_accumulate(m, inp, tgt, seq)
    errs = tap_errors(m, e, cfg, 2, FWD_TAPS + BWD_TAPS)
    assert max(errs.values()) < F32_TOL, max(errs.items(), key=lambda kv: kv[1])
    rep = []
    assert compare_grads(m, e, rep) < F32_TOL, rep
    e.close()


@pytest.mark.parametrize("arch,hd,heads,kv,seq", [
    (O.ARCH_L, 32, 2, 1, 256), (O.ARCH_L, 40, 2, 2, 193), (O.ARCH_L, 48, 4, 2, 255), (O.ARCH_L, 64, 2, 1, 257), (O.ARCH_N, 64, 2, 2, 256)])
def test_fp32_tiles_of_several_sweeps(arch, hd, heads, kv, seq):
    """Up to 256 positions the dQ kernel keeps the scores of all its tiles; from 257 on it forms them twice."""
    test_fp32_tiles(arch, hd, heads, kv, seq)


@pytest.mark.parametrize("hd,heads,kv,seq,batch", [
    (32, 4, 4, 65, 49), (32, 4, 4, 65, 70), (40, 2, 2, 193, 50), (64, 2, 2, 64, 150), (64, 2, 1, 129, 80), (64, 2, 2, 256, 37), (64, 2, 2, 256, 38)])
def test_fp32_tiles_of_many_blocks(hd, heads, kv, seq, batch):
    """More blocks than the SMs hold with two buffers take one, more than four an SM with four tiles of head size 64, or two of 32, two sweeps for dQ."""
    cfg, m, e, inp, tgt = _step(ane.DTYPE_F32, O.ARCH_L, 0, hd, heads, kv, seq, batch, 0.1)
    oracle_batch_accumulate(m, inp, tgt, seq)
    rep = []
    assert compare_grads(m, e, rep) < F32_TOL, rep
    e.close()


@pytest.mark.parametrize("hd,heads,kv,seq,batch", [(32, 2, 1, 63, 2), (48, 2, 2, 65, 2), (48, 4, 2, 200, 2), (48, 2, 2, 257, 50),
                                                   (64, 2, 1, 100, 2), (64, 4, 4, 129, 40)])
def test_bf16_tiles(hd, heads, kv, seq, batch):
    """q, k, v and d att are rounded to bf16 (2^-9 each) before products that cancel: dq / dk within 2e-2 as the
    kernels for head size 64 (test_bf16_attention_multi_tile_sequences), everything forward within 1e-2."""
    cfg, m, e, inp, tgt = _step(ane.DTYPE_BF16, O.ARCH_L, 0, hd, heads, kv, seq, batch, 0.05)
    m.accumulate(np.ascontiguousarray(inp[-1]), np.ascontiguousarray(tgt[-1]))  # the oracle's taps are its last sequence's
    for layer in range(cfg["layers"]):
        for tap, tol in ((O.TAP_Q, 1e-2), (O.TAP_ATT, 1e-2), (O.TAP_DQ, 2e-2), (O.TAP_DK, 2e-2), (O.TAP_DV, 2e-2)):
            want = m.tap(tap, layer).astype(np.float64)
            got = e.tap(tap, layer).reshape(batch, want.shape[0], seq)[-1].astype(np.float64)
            err = np.linalg.norm(got - want) / np.linalg.norm(want)
            assert err < tol, (layer, tap, err)
    e.close()


@pytest.mark.parametrize("hd", [48, 64])
def test_more_heads_than_a_grid_dimension_takes(hd):
    """33000 windows of two tokens with two heads: 66000 heads in one launch.  Every window is the same, and so must be its
    attention output and gradients."""
    batch, seq, heads = 33000, 2, 2
    e = ane.open(ane.Options(dim=hd * heads, hidden=32, n_layers=1, n_heads=heads, n_kv_heads=heads, vocab=96, seq=seq, batch=batch,
                             arch=ane.ARCH_LLAMA, quirks=0, compute_dtype=ane.DTYPE_BF16, accum_steps=1000, debug_taps=True))
    rng = np.random.default_rng(2)
    for tid, layer in ((ane.T_EMBED, 0), (ane.T_WQ, 0), (ane.T_WK, 0), (ane.T_WV, 0), (ane.T_WO, 0)):
        e.import_tensor(tid, layer, (0.2 * rng.standard_normal(e.tensor_size(tid, layer))).astype(np.float32))
    toks = np.tile(np.array([3, 7], np.uint16), (batch, 1))
    r = e.step_tokens(toks, toks[:, ::-1].copy())
    assert r.device_status == 0 and np.isfinite(r.loss)
    for tap in (O.TAP_ATT, O.TAP_DQ, O.TAP_DK, O.TAP_DV):
        out = e.tap(tap, 0).reshape(batch, -1)
        assert np.abs(out[0]).max() > 0
        np.testing.assert_array_equal(out, np.broadcast_to(out[0], out.shape))
    e.close()


def _bf16(x):
    """float64 -> nearest bf16, as float64."""
    u = np.asarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return (((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16).astype(np.uint32).view(np.float32).astype(np.float64)


def attention_error_over_rounding(hd, heads, kv, seq, batch, std):
    """{tensor: error of the engine's attention / the error that rounding the exact result to bf16 makes}, where exact is
    attention in float64 on the engine's own bf16 operands (Wo = 1, so that d att is bf16(d x2))."""
    cfg, m, e, inp, tgt = _step(ane.DTYPE_BF16, O.ARCH_L, 0, hd, heads, kv, seq, batch, std)
    e.import_tensor(ane.T_WO, 0, np.eye(hd * heads, dtype=np.float32))
    e.import_tensor(ane.T_WO, 1, np.eye(hd * heads, dtype=np.float32))
    e.step_tokens(inp, tgt)
    tap = lambda t, h: e.tap(t, 0).reshape(batch, h, hd, seq).astype(np.float64).transpose(0, 1, 3, 2)  # noqa: E731
    q, k, v, do = tap(O.TAP_Q, heads), tap(O.TAP_K, kv), tap(O.TAP_V, kv), _bf16(tap(O.TAP_DX2, heads))
    got = {"att": tap(O.TAP_ATT, heads), "dq": tap(O.TAP_DQ, heads), "dk": tap(O.TAP_DK, kv), "dv": tap(O.TAP_DV, kv)}
    e.close()
    rep = heads // kv
    kr, vr = k.repeat(rep, 1), v.repeat(rep, 1)
    s = q @ kr.transpose(0, 1, 3, 2) / np.sqrt(hd)
    s[..., np.triu(np.ones((seq, seq), bool), 1)] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    dp = do @ vr.transpose(0, 1, 3, 2)
    ds = p * (dp - (p * dp).sum(-1, keepdims=True)) / np.sqrt(hd)
    shared = lambda x: x.reshape(batch, kv, rep, seq, hd).sum(2)  # noqa: E731
    want = {"att": p @ vr, "dq": ds @ kr, "dk": shared(ds.transpose(0, 1, 3, 2) @ q), "dv": shared(p.transpose(0, 1, 3, 2) @ do)}
    angle = np.arange(seq)[:, None] * 10000.0 ** (-np.arange(0, hd, 2) / hd)
    c, sn = np.cos(angle), np.sin(angle)
    for name in ("dq", "dk"):  # the rotation undone
        x, y = want[name][..., ::2].copy(), want[name][..., 1::2].copy()
        want[name][..., ::2], want[name][..., 1::2] = x * c + y * sn, y * c - x * sn
    return {n: np.linalg.norm(got[n] - want[n]) / np.linalg.norm(_bf16(want[n]) - want[n]) for n in got}


@pytest.mark.parametrize("hd,heads,kv,seq,batch", [(32, 2, 1, 63, 2), (48, 2, 2, 65, 2), (48, 4, 2, 200, 2), (48, 2, 2, 257, 50)])
@pytest.mark.parametrize("std", [0.02, 0.15])
def test_probabilities_keep_sixteen_bits(hd, heads, kv, seq, batch, std):
    """Probabilities and score gradients enter their products as bf16 hi + lo (2^-17 each), so that the result is off by its
    own rounding (2^-9) and little else: 2 % more is 2^-9 sqrt(1.02^2 - 1) = 2^-11.3 of the result, ten times what their
    2^-17 and the 2^-17 of delta's O leave after the differences they enter.  Rounded to bf16 alone they exceed it."""
    off = attention_error_over_rounding(hd, heads, kv, seq, batch, std)
    assert max(off.values()) < 1.02, off
