"""tcgen05 GEMM (and fp32 products on the FMA units and the tensor cores) against the oracle's naive loops, through the C ABI.
Shapes cover the step's three operand layouts, ragged edges and split-K accumulation."""
import ctypes

import numpy as np
import pytest

import ane
from ane import _ffi
from oracle import oracle as O
from parity_utils import rel_l2

pytestmark = pytest.mark.gpu
lib = _ffi.lib


def _ck(rc):
    assert rc == 0, lib.ane_ops_last_error().decode()


def _up(a):
    a = np.ascontiguousarray(a, dtype=np.float32)
    p = lib.ane_dev_malloc(a.nbytes)
    _ck(lib.ane_dev_h2d(p, a.ctypes.data, a.nbytes))
    return p


def _up_bf16(a):
    p = _up(a)
    q = lib.ane_dev_malloc(a.size * 2)
    _ck(lib.ane_op_cast_f32_to_bf16(p, q, a.size))
    lib.ane_dev_free(p)
    return q


def _down(p, shape):
    a = np.empty(shape, dtype=np.float32)
    _ck(lib.ane_dev_d2h(a.ctypes.data, p, a.nbytes))
    return a


def _bf16_round(a):
    u = np.ascontiguousarray(a, dtype=np.float32).view(np.uint32).astype(np.uint64)
    r = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16) << 16
    return r.astype(np.uint32).view(np.float32).reshape(a.shape)


def _fp(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_float))


def _gemm(dtype, A_store, B_store, C_init, M, N, K, a_mn, b_mn, out_mode, split_k=0, res=None):
    upf = _up_bf16 if dtype == ane.DTYPE_BF16 else _up
    dA, dB, dC = upf(A_store), upf(B_store), _up(C_init)
    dR = _up(res) if res is not None else None
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype = dtype
    g.d_a, g.d_b, g.d_c = dA, dB, dC
    g.m, g.n, g.k = M, N, K
    g.lda, g.ldb, g.ldc = A_store.shape[1], B_store.shape[1], N
    g.a_mn, g.b_mn, g.out_mode, g.alpha, g.split_k = a_mn, b_mn, out_mode, 1.0, split_k
    if dR is not None:
        g.d_res1, g.ldres = dR, N
    _ck(lib.ane_op_gemm(ctypes.byref(g)))
    _ck(lib.ane_dev_sync())
    st = ctypes.c_int32(0)
    _ck(lib.ane_ops_device_status(ctypes.byref(st)))
    assert st.value == 0
    out = _down(dC, (M, N))
    for p in (dA, dB, dC) + ((dR,) if dR is not None else ()):
        lib.ane_dev_free(p)
    return out


def test_step_sized_shapes_take_the_wide_tile_and_tma_residual_paths():
    """Shapes of the 110M step that select the 256-row tiles (long K, enough tiles), the stream-K weight
    gradient on 256-row tiles and the TMA-fed residual epilogue; checked against numpy on the same
    bf16-rounded operands (fp32 accumulation order differs, hence 1e-4)."""
    rng = np.random.default_rng(3)
    # dx form: C[M,N] = A[M,K] . B[K,N]
    M, N, K = 8192, 768, 2304
    A = _bf16_round(rng.standard_normal((M, K)).astype(np.float32) * 0.1)
    B = _bf16_round(rng.standard_normal((K, N)).astype(np.float32) * 0.1)
    got = _gemm(ane.DTYPE_BF16, A, B, np.zeros((M, N), np.float32), M, N, K, 0, 1, 1)
    assert rel_l2(got, A @ B) < 1e-4
    # dW form with accumulation: C[M,N] += A^T[M,K] . B[K,N], A stored [K, M]
    M, N, K = 2304, 768, 8192
    At = _bf16_round(rng.standard_normal((K, M)).astype(np.float32) * 0.1)
    B = _bf16_round(rng.standard_normal((K, N)).astype(np.float32) * 0.1)
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    got = _gemm(ane.DTYPE_BF16, At, B, C0, M, N, K, 1, 1, 2)
    assert rel_l2(got, C0 + At.T @ B) < 1e-4
    # forward form with a residual: C = A . W^T + R
    M, N, K = 8192, 768, 768
    A = _bf16_round(rng.standard_normal((M, K)).astype(np.float32) * 0.1)
    W = _bf16_round(rng.standard_normal((N, K)).astype(np.float32) * 0.1)
    R = rng.standard_normal((M, N)).astype(np.float32)
    got = _gemm(ane.DTYPE_BF16, A, W, np.zeros((M, N), np.float32), M, N, K, 0, 0, 1, res=R)
    assert rel_l2(got, A @ W.T + R) < 1e-4
    # ragged rows and columns through the same residual path (TMA clips the residual pieces)
    M, N, K = 8100, 760, 768
    got = _gemm(ane.DTYPE_BF16, A[:M], W[:N], np.zeros((M, N), np.float32), M, N, K, 0, 0, 1, res=np.ascontiguousarray(R[:M, :N]))
    assert rel_l2(got, A[:M] @ W[:N].T + R[:M, :N]) < 1e-4


def test_short_k_wide_n_shapes_take_the_cta_pair_tiles():
    """K = 768 with enough 256 x 256 tiles to fill the CTA pairs: the planner picks the two-CTA kernel
    (tcgen05.mma.cta_group::2, half of the B tile per CTA).  Both B layouts, a residual, and ragged M and N
    (the second CTA's rows / B columns then start or end outside the tensors)."""
    rng = np.random.default_rng(5)
    for (M, N, K, b_mn, res) in [(8192, 2304, 768, 0, False), (4000, 2300, 768, 1, False), (3900, 2304, 704, 0, True),
                                 (8192, 2048, 768, 1, False)]:
        A = _bf16_round(rng.standard_normal((M, K)).astype(np.float32) * 0.1)
        if b_mn:
            B = _bf16_round(rng.standard_normal((K, N + (-N) % 8)).astype(np.float32) * 0.1)   # 16-byte row pitch
            want = A @ B[:, :N]
        else:
            B = _bf16_round(rng.standard_normal((N, K)).astype(np.float32) * 0.1)
            want = A @ B.T
        R = rng.standard_normal((M, N)).astype(np.float32) if res else None
        got = _gemm(ane.DTYPE_BF16, A, B, np.zeros((M, N), np.float32), M, N, K, 0, b_mn, 1, res=R)
        assert rel_l2(got, want + (R if res else 0)) < 1e-4, (M, N, K, b_mn, res)


def test_split_precision_gemm_carries_fp32_operands_through_the_tensor_cores():
    """ANE_DTYPE_BF16X3: fp32 operands cut into bf16 (hi, lo) pairs, three tcgen05 products.  Against float64
    on the unrounded operands the result must be fp32-like (a single bf16 product is ~3e-3 off); the three
    operand layouts of the step, a residual, an accumulating output and ragged sizes."""
    rng = np.random.default_rng(8)
    M, N, K = 1024, 768, 2304
    A = rng.standard_normal((M, K)).astype(np.float32)
    B = rng.standard_normal((K, N)).astype(np.float32)
    got = _gemm(ane.DTYPE_BF16X3, A, B, np.zeros((M, N), np.float32), M, N, K, 0, 1, 1)
    want = A.astype(np.float64) @ B.astype(np.float64)
    assert rel_l2(got, want) < 2e-5
    one = _gemm(ane.DTYPE_BF16, A, B, np.zeros((M, N), np.float32), M, N, K, 0, 1, 1)
    assert rel_l2(one, want) > 1e-3                                     # the single bf16 product, for scale
    M, N, K = 1000, 760, 776                                            # forward form, ragged, with a residual
    A = rng.standard_normal((M, K)).astype(np.float32)
    W = rng.standard_normal((N, K)).astype(np.float32)
    R = rng.standard_normal((M, N)).astype(np.float32)
    got = _gemm(ane.DTYPE_BF16X3, A, W, np.zeros((M, N), np.float32), M, N, K, 0, 0, 1, res=R)
    assert rel_l2(got, A.astype(np.float64) @ W.astype(np.float64).T + R) < 2e-5
    M, N, K = 2304, 768, 2048                                           # weight-gradient form, accumulating
    At = rng.standard_normal((K, M)).astype(np.float32)
    B = rng.standard_normal((K, N)).astype(np.float32)
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    got = _gemm(ane.DTYPE_BF16X3, At, B, C0, M, N, K, 1, 1, 2)
    assert rel_l2(got, C0 + At.astype(np.float64).T @ B.astype(np.float64)) < 2e-5


@pytest.mark.parametrize("b_mn", [0, 1])
@pytest.mark.parametrize("n,k", [(768, 768), (2304, 768), (768, 2048), (768, 2304)])
def test_split_precision_rows_do_not_depend_on_the_number_of_rows(b_mn, n, k):
    """A split-precision product has one accumulator for the whole contraction, whatever tiles there are beside it: the rows of
    a small product are those of a large one, bit for bit."""
    rng = np.random.default_rng(n + k)
    A = rng.standard_normal((4096, k)).astype(np.float32)
    B = rng.standard_normal((k, n) if b_mn else (n, k)).astype(np.float32)
    large = _gemm(ane.DTYPE_BF16X3, A, B, np.zeros((4096, n), np.float32), 4096, n, k, 0, b_mn, 1)
    for m in (100, 256, 512):
        small = _gemm(ane.DTYPE_BF16X3, A[:m], B, np.zeros((m, n), np.float32), m, n, k, 0, b_mn, 1)
        np.testing.assert_array_equal(small, large[:m])


@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1), (1, 0)])
@pytest.mark.parametrize("m,n,k", [(128, 96, 16), (4, 4, 4), (100, 92, 60), (288, 96, 2048), (97 * 4, 132, 1000), (2048, 288, 288), (20000, 128, 36)])
def test_fp32_tiles_and_cluster_splits(a_mn, b_mn, m, n, k):
    """96- and 128-wide tiles, one block and clusters of 2, 4 and 8 along the contraction, ragged edges, a residual and
    accumulation.  Any order of k fp32 additions of N(0, 1) products is within sqrt(k) 2^-23 < 1e-5 (rel-L2)."""
    rng = np.random.default_rng(m + n + k)
    A = rng.standard_normal((m, k)).astype(np.float32)
    B = rng.standard_normal((k, n)).astype(np.float32)
    C = rng.standard_normal((m, n)).astype(np.float32)
    a = np.ascontiguousarray(A.T) if a_mn else A
    b = B if b_mn else np.ascontiguousarray(B.T)
    want = A.astype(np.float64) @ B.astype(np.float64) + C
    assert rel_l2(_gemm(ane.DTYPE_F32, a, b, np.zeros_like(C), m, n, k, a_mn, b_mn, 1, res=C), want) < 1e-5
    assert rel_l2(_gemm(ane.DTYPE_F32, a, b, C, m, n, k, a_mn, b_mn, 2), want) < 1e-5


@pytest.mark.parametrize("dtype", [ane.DTYPE_BF16, ane.DTYPE_F32, ane.DTYPE_BF16X3])
@pytest.mark.parametrize("oc,ic,seq", [(96, 64, 40), (256, 136, 300), (768, 256, 128)])
def test_linear_forward_dx_dw_match_oracle(dtype, oc, ic, seq):
    """linearCF / linearBackwardDXCF / accumLinearGradCF (ane/common.go:91, ane/train_full.go:213,242)."""
    rng = np.random.default_rng(oc + seq)
    rnd = _bf16_round if dtype == ane.DTYPE_BF16 else (lambda a: a)
    W = rnd(rng.standard_normal((oc, ic)).astype(np.float32) * 0.1)
    x_cf = rnd(rng.standard_normal((ic, seq)).astype(np.float32))          # reference layout [C][seq]
    dy_cf = rnd(rng.standard_normal((oc, seq)).astype(np.float32))
    tol = 2e-5
    # forward: y[t,o] = x[t,:] . W[o,:]
    want = np.empty((oc, seq), np.float32)
    O.lib().orc_linear(_fp(want), _fp(W), _fp(x_cf), oc, ic, seq)
    got = _gemm(dtype, np.ascontiguousarray(x_cf.T), W, np.zeros((seq, oc), np.float32), seq, oc, ic, 0, 0, 1)
    assert rel_l2(got.T, want) < tol
    # dx[t,i] = dy[t,:] . W[:,i]   (B stored [K=oc, N=ic])
    want = np.empty((ic, seq), np.float32)
    O.lib().orc_linear_dx(_fp(want), _fp(W), _fp(dy_cf), oc, ic, seq)
    got = _gemm(dtype, np.ascontiguousarray(dy_cf.T), W, np.zeros((seq, ic), np.float32), seq, ic, oc, 0, 1, 1)
    assert rel_l2(got.T, want) < tol
    # dW[o,i] += sum_t dy[t,o] x[t,i]   (both operands stored [K=seq, .]); beta = 1
    dw0 = rng.standard_normal((oc, ic)).astype(np.float32)
    want = dw0.copy()
    O.lib().orc_linear_dw(_fp(want), _fp(dy_cf), _fp(x_cf), oc, ic, seq)
    for split in (1, 2):
        got = _gemm(dtype, np.ascontiguousarray(dy_cf.T), np.ascontiguousarray(x_cf.T), dw0, oc, ic, seq, 1, 1, 2, split)
        assert rel_l2(got, want) < tol


def _down_bf16(p, shape):
    n = int(np.prod(shape))
    q = lib.ane_dev_malloc(n * 4)
    _ck(lib.ane_op_cast_bf16_to_f32(p, q, n))
    out = _down(q, shape)
    lib.ane_dev_free(q)
    return out


@pytest.mark.parametrize("M,Hd,K", [(8192, 2048, 768), (300, 96, 136), (1000, 2048, 768)])
def test_swiglu_backward_fused_into_the_dx_product(M, Hd, K):
    """out_mode 7: d gate = dOut . W2 stays in the accumulators; the epilogue reads h1 | h3 (interleaved in blocks
    of 32 columns) and writes d h1 = d gate * h3 * silu'(h1), d h3 = d gate * silu(h1) in the same layout.  Against
    float64 on the same bf16 operands; the step's shape (CTA-pair tiles) and ragged ones (single-CTA tiles)."""
    rng = np.random.default_rng(M + Hd)
    dOut = _bf16_round(rng.standard_normal((M, K)).astype(np.float32))
    W2 = _bf16_round((rng.standard_normal((K, Hd)) / np.sqrt(K)).astype(np.float32))       # stored [K, N]: MN-major B
    h1 = _bf16_round(rng.standard_normal((M, Hd)).astype(np.float32) * 2.0)
    h3 = _bf16_round(rng.standard_normal((M, Hd)).astype(np.float32))
    h13 = np.empty((M, 2 * Hd), np.float32)
    blk = h13.reshape(M, Hd // 32, 2, 32)
    blk[:, :, 0, :] = h1.reshape(M, Hd // 32, 32)
    blk[:, :, 1, :] = h3.reshape(M, Hd // 32, 32)
    dA, dB, dH = _up_bf16(dOut), _up_bf16(W2), _up_bf16(h13)
    dC = lib.ane_dev_malloc(M * 2 * Hd * 2)
    _ck(lib.ane_dev_memset(dC, 0xFF, M * 2 * Hd * 2))
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype = ane.DTYPE_BF16
    g.d_a, g.d_b, g.d_c, g.d_aux = dA, dB, dC, dH
    g.m, g.n, g.k = M, Hd, K
    g.lda, g.ldb, g.ldc, g.ldaux = K, Hd, 2 * Hd, 2 * Hd
    g.a_mn, g.b_mn, g.out_mode, g.alpha = 0, 1, 7, 1.0
    _ck(lib.ane_op_gemm(ctypes.byref(g)))
    _ck(lib.ane_dev_sync())
    st = ctypes.c_int32(0)
    _ck(lib.ane_ops_device_status(ctypes.byref(st)))
    assert st.value == 0
    got = _down_bf16(dC, (M, 2 * Hd)).reshape(M, Hd // 32, 2, 32)
    dg = dOut.astype(np.float64) @ W2.astype(np.float64)
    x = h1.astype(np.float64)
    sg = 1.0 / (1.0 + np.exp(-x))
    want1 = dg * h3 * sg * (1.0 + x * (1.0 - sg))
    want3 = dg * x * sg
    assert np.isfinite(got).all()
    assert rel_l2(got[:, :, 0, :].reshape(M, Hd), want1) < 4e-3          # one bf16 rounding of the output
    assert rel_l2(got[:, :, 1, :].reshape(M, Hd), want3) < 4e-3
    for p in (dA, dB, dH, dC):
        lib.ane_dev_free(p)


@pytest.mark.parametrize("M,Hd,K", [(8192, 2048, 768), (320, 192, 128), (100, 64, 72)])
def test_relu2_backward_fused_into_the_dx_product(M, Hd, K):
    """out_mode 10: d gate = dOut . W2 stays in the accumulators; the epilogue reads h and writes
    d h = d gate * 2 max(h, 0) (the reference's ReLU^2 activation, ane/common.go:146, differentiated).  Against
    float64 on the same bf16 operands; the step's shape (CTA-pair tiles) and ragged ones (single-CTA tiles)."""
    rng = np.random.default_rng(M + Hd + 1)
    dOut = _bf16_round(rng.standard_normal((M, K)).astype(np.float32))
    W2 = _bf16_round((rng.standard_normal((K, Hd)) / np.sqrt(K)).astype(np.float32))       # stored [K, N]: MN-major B
    h = _bf16_round(rng.standard_normal((M, Hd)).astype(np.float32) * 2.0)
    dA, dB, dH = _up_bf16(dOut), _up_bf16(W2), _up_bf16(h)
    dC = lib.ane_dev_malloc(M * Hd * 2)
    _ck(lib.ane_dev_memset(dC, 0xFF, M * Hd * 2))
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype = ane.DTYPE_BF16
    g.d_a, g.d_b, g.d_c, g.d_aux = dA, dB, dC, dH
    g.m, g.n, g.k = M, Hd, K
    g.lda, g.ldb, g.ldc, g.ldaux = K, Hd, Hd, Hd
    g.a_mn, g.b_mn, g.out_mode, g.alpha = 0, 1, 10, 1.0
    _ck(lib.ane_op_gemm(ctypes.byref(g)))
    _ck(lib.ane_dev_sync())
    st = ctypes.c_int32(0)
    _ck(lib.ane_ops_device_status(ctypes.byref(st)))
    assert st.value == 0
    got = _down_bf16(dC, (M, Hd))
    want = (dOut.astype(np.float64) @ W2.astype(np.float64)) * 2.0 * np.maximum(h.astype(np.float64), 0.0)
    assert np.isfinite(got).all()
    assert rel_l2(got, want) < 4e-3          # one bf16 rounding of the output
    assert np.all(got[h <= 0] == 0)          # exact zeros where the activation was off
    for p in (dA, dB, dH, dC):
        lib.ane_dev_free(p)


@pytest.mark.parametrize("M,N,K,b_mn", [(1, 8, 256, 0), (37, 768, 768, 0), (128, 128, 1024, 1), (256, 768, 4096, 1), (129, 136, 520, 0),
                                        (300, 2304, 768, 0), (512, 1000, 264, 1)])
def test_products_of_few_tiles(M, N, K, b_mn):
    """Less than a wave of 128 x 128 tiles: 32- and 64-column ones, ragged rows and columns, plain and with a residual that TMA feeds or the
    threads read."""
    rng = np.random.default_rng(M + N + K)
    A = _bf16_round(rng.standard_normal((M, K)).astype(np.float32) * 0.1)
    B = _bf16_round(rng.standard_normal((K, N) if b_mn else (N, K)).astype(np.float32) * 0.1)
    R = rng.standard_normal((M, N)).astype(np.float32)
    want = A.astype(np.float64) @ (B if b_mn else B.T).astype(np.float64)
    assert rel_l2(_gemm(ane.DTYPE_BF16, A, B, np.zeros((M, N), np.float32), M, N, K, 0, b_mn, 1), want) < 1e-5
    assert rel_l2(_gemm(ane.DTYPE_BF16, A, B, np.zeros((M, N), np.float32), M, N, K, 0, b_mn, 1, res=R), want + R) < 1e-5


@pytest.mark.parametrize("M,Hd,K", [(256, 2048, 768), (200, 320, 264), (100, 64, 512)])
def test_activation_backward_on_narrow_tiles(M, Hd, K):
    """Few enough tiles for 64-column ones, whose epilogues keep one input piece in flight, or two (SwiGLU)."""
    test_swiglu_backward_fused_into_the_dx_product(M, Hd, K)
    test_relu2_backward_fused_into_the_dx_product(M, Hd, K)


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,out", [(1, 8, 72, 0, 0, 1), (129, 72, 520, 0, 0, 1), (256, 768, 2048, 0, 0, 1), (300, 40, 64, 0, 0, 0),
                                                 (256, 2304, 768, 0, 0, 0), (200, 136, 520, 0, 1, 1), (256, 768, 768, 0, 1, 0),
                                                 (136, 72, 200, 1, 1, 2), (768, 768, 256, 1, 1, 2)])
def test_narrow_tiles_give_the_sums_of_wide_ones(M, N, K, a_mn, b_mn, out):
    """Products with few tiles run on 64- or 32-column tiles (fp32 store, bf16 store, accumulation): against float64, and bit for bit
    the same as those rows of a product large enough for wide tiles."""
    rng = np.random.default_rng(M + N + K + out)
    big = 32768 if a_mn else 8192
    A = _bf16_round(rng.standard_normal((K, big) if a_mn else (big, K)).astype(np.float32) * 0.1)
    B = _bf16_round(rng.standard_normal((K, N) if b_mn else (N, K)).astype(np.float32) * 0.1)
    few = np.ascontiguousarray(A[:, :M] if a_mn else A[:M])
    C = np.ones((big, N), np.float32)
    run = lambda a, m: _bf16_result(a, B, m, N, K, b_mn) if out == 0 else _gemm(ane.DTYPE_BF16, a, B, C[:m], m, N, K, a_mn, b_mn, out)  # noqa: E731
    got = run(few, M)
    want = (few.T if a_mn else few).astype(np.float64) @ (B if b_mn else B.T).astype(np.float64) + (1.0 if out == 2 else 0.0)
    assert rel_l2(got, want) < (4e-3 if out == 0 else 1e-5)
    np.testing.assert_array_equal(got, run(A, big)[:M])


def _bf16_result(A, B, M, N, K, b_mn):
    dA, dB, dC = _up_bf16(A), _up_bf16(B), lib.ane_dev_malloc(M * N * 2)
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype = ane.DTYPE_BF16
    g.d_a, g.d_b, g.d_c = dA, dB, dC
    g.m, g.n, g.k, g.lda, g.ldb, g.ldc = M, N, K, K, N if b_mn else K, N
    g.b_mn, g.out_mode, g.alpha = b_mn, 0, 1.0
    _ck(lib.ane_op_gemm(ctypes.byref(g)))
    got = _down_bf16(dC, (M, N))
    for p in (dA, dB, dC):
        lib.ane_dev_free(p)
    return got


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,out", [(513, 4096, 136, 0, 0, 1), (1025, 1000, 288, 0, 1, 1), (2048, 288, 768, 0, 0, 1), (1000, 2304, 264, 1, 0, 1),
                                                 (864, 288, 2048, 1, 1, 2), (520, 264, 8200, 1, 1, 2), (2048, 288, 4096, 0, 1, 1)])
def test_fp32_products_on_the_tensor_cores(M, N, K, a_mn, b_mn, out):
    """Large fp32 products (all of these sizes) run as six products of bf16 parts, whole tiles and tiles shared by a cluster, with residuals and as
    accumulation.  The error of a sum of K fp32 products in any order is about sqrt(K) / 2 roundings of 2^-24 in the 2-norm;
    held to a quarter of that, and for terms of one sign to 2^-23.  Elements that an infinite or NaN operand touches are what fp32 FMAs give."""
    rng = np.random.default_rng(M + N + K)
    for positive in (False, True):
        draw = (lambda *s: rng.random(s, dtype=np.float32)) if positive else (lambda *s: rng.standard_normal(s, dtype=np.float32))  # noqa: E731
        A, B, R = draw(*((K, M) if a_mn else (M, K))), draw(*((K, N) if b_mn else (N, K))), draw(M, N)
        want = (A.T if a_mn else A).astype(np.float64) @ (B if b_mn else B.T).astype(np.float64)
        got = _gemm(ane.DTYPE_F32, A, B, R, M, N, K, a_mn, b_mn, 2) if out == 2 else _gemm(ane.DTYPE_F32, A, B, np.zeros_like(R), M, N, K, a_mn, b_mn, 1, res=R)
        assert rel_l2(got, want + R) < (2.0**-23 if positive else max(np.sqrt(K) / 8, 2.0) * 2.0**-24)
    # One term per sum: the FMA units would round the product of the two operands once, parts that are added and cut off are a bit off here and there.
    one = np.zeros_like(A)
    term = np.arange(M) % K
    (one.T if a_mn else one)[np.arange(M), term] = draw(M)
    exact = (one.T if a_mn else one)[np.arange(M), term][:, None] * (B if b_mn else B.T)[term]
    got = _gemm(ane.DTYPE_F32, one, B, np.zeros_like(R), M, N, K, a_mn, b_mn, out)
    assert (got != exact).any()
    np.testing.assert_allclose(got, exact, rtol=2.0**-22)
    at = (A.T if a_mn else A), (B if b_mn else B.T)  # views: [M, K] and [K, N]
    at[0][3, 5], at[0][7, 1], at[1][4, 2], at[0][9, 0] = np.inf, np.nan, -np.inf, 3.4e38
    with np.errstate(invalid="ignore", over="ignore"):
        want = np.vstack([at[0][r].astype(np.float64) @ at[1].astype(np.float64) for r in (3, 7, 9, 11)]).astype(np.float32)
    got = _gemm(ane.DTYPE_F32, A, B, np.zeros_like(R), M, N, K, a_mn, b_mn, out)[[3, 7, 9, 11]]
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    far = ~np.isfinite(want)
    np.testing.assert_array_equal(got[far], want[far])
    np.testing.assert_allclose(got[~far], want[~far], rtol=1e-4)


@pytest.mark.parametrize("M,N,K,a_mn,b_mn,out", [(1025, 1000, 288, 0, 1, 1), (864, 288, 2048, 1, 1, 2), (520, 264, 8200, 0, 0, 1)])
def test_fp32_products_keep_their_precision_over_the_range_of_fp32(M, N, K, a_mn, b_mn, out):
    """Operands far from one, down to subnormal ones and up to where products overflow, have the error bound of those around one (see above); sums
    that are formed again, K / 32 terms a lane, stay below it.  Products of powers of two scale exactly, so the reference does too."""
    rng = np.random.default_rng(M + K)
    A, B = rng.standard_normal((K, M) if a_mn else (M, K)), rng.standard_normal((K, N) if b_mn else (N, K))
    for ea, eb in ((-115, 40), (40, -122), (-130, 60), (-146, 90), (-60, -60), (60, 50), (118, -100), (-20, 123)):
        a, b = (A * 2.0**ea).astype(np.float32), (B * 2.0**eb).astype(np.float32)
        want = (np.ldexp(a.astype(np.float64), -ea).T if a_mn else np.ldexp(a.astype(np.float64), -ea)) @ (np.ldexp(b.astype(np.float64), -eb) if b_mn else np.ldexp(b.astype(np.float64), -eb).T)
        got = np.ldexp(_gemm(ane.DTYPE_F32, a, b, np.zeros((M, N), np.float32), M, N, K, a_mn, b_mn, out).astype(np.float64), -ea - eb)
        assert rel_l2(got, want) < max(np.sqrt(K) / 8, 2.0) * 2.0**-24, (ea, eb)


@pytest.mark.parametrize("M,N,K,a_mn,b_mn", [(2048, 1544, 4096, 0, 0), (2048, 1544, 4096, 0, 1), (520, 264, 8200, 1, 1), (520, 264, 8200, 1, 0)])
def test_fp32_products_of_nan_and_infinities_cost_about_what_finite_ones_do(M, N, K, a_mn, b_mn):
    """Sums that the tensor cores leave NaN are formed again; a whole operand of NaN and a row of infinities, on more tiles than SMs and on
    tiles shared by a cluster.  One thread per sum to the end of the contraction took 50 times as long as finite numbers, and ever longer with K."""
    rng = np.random.default_rng(M + K)
    A, B = rng.random((K, M) if a_mn else (M, K), dtype=np.float32), rng.random((K, N) if b_mn else (N, K), dtype=np.float32)
    row = A.copy()
    (row.T if a_mn else row)[77] = np.inf
    dB, dC = _up(B), _up(np.zeros((M, N), np.float32))
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype, g.d_b, g.d_c = ane.DTYPE_F32, dB, dC
    g.m, g.n, g.k, g.lda, g.ldb, g.ldc = M, N, K, A.shape[1], B.shape[1], N
    g.a_mn, g.b_mn, g.out_mode, g.alpha = a_mn, b_mn, 1, 1.0
    times, results = [], []
    for a in (A, np.full_like(A, np.nan), row):
        g.d_a = _up(a)
        took = []
        for _ in range(4):
            ms = ctypes.c_float(0)
            _ck(lib.ane_timer_begin())
            _ck(lib.ane_op_gemm(ctypes.byref(g)))
            _ck(lib.ane_timer_end(ctypes.byref(ms)))
            took.append(ms.value)
        st = ctypes.c_int32(0)
        _ck(lib.ane_ops_device_status(ctypes.byref(st)))
        assert st.value == 0
        times.append(min(took))
        results.append(_down(dC, (M, N)))
        lib.ane_dev_free(g.d_a)
    lib.ane_dev_free(dB)
    lib.ane_dev_free(dC)
    assert np.isnan(results[1]).all()
    assert (results[2][77] == np.inf).all()
    np.testing.assert_array_equal(np.delete(results[2], 77, 0), np.delete(results[0], 77, 0))
    assert times[1] < 8 * times[0] and times[2] < 8 * times[0], times


def test_fp32_products_are_queued_without_waiting_or_allocating():
    """A large fp32 product beside a sleeping stream returns at once, as the other products do, also by two threads with operands of their own, and
    does not disturb what another stream of the thread captures."""
    import threading

    import torch
    M, N, K = 1024, 768, 768
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    jobs = []
    for _ in range(2):
        a, b = torch.randn(M, K, device="cuda", generator=gen), torch.randn(N, K, device="cuda", generator=gen)
        c = torch.zeros(M, N, device="cuda")
        g = _ffi.GemmArgs()
        g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
        g.dtype, g.d_a, g.d_b, g.d_c = ane.DTYPE_F32, a.data_ptr(), b.data_ptr(), c.data_ptr()
        g.m, g.n, g.k, g.lda, g.ldb, g.ldc, g.out_mode, g.alpha = M, N, K, K, K, N, 1, 1.0
        _ck(lib.ane_op_gemm(ctypes.byref(g)))
        jobs.append((g, a, b, c, c.clone()))
    torch.cuda.synchronize()
    for _, a, b, _, first in jobs:
        assert rel_l2(first.cpu().numpy(), (a.double() @ b.double().T).cpu().numpy()) < 4e-7
    torch.cuda._sleep(200_000_000)  # about 0.1 s on the default stream
    for g, *_ in jobs:
        _ck(lib.ane_op_gemm(ctypes.byref(g)))
    assert not torch.cuda.current_stream().query()
    torch.cuda.synchronize()

    def many(g, a, b, c, first):
        for _ in range(50):
            lib.ane_op_gemm(ctypes.byref(g))

    threads = [threading.Thread(target=many, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for _, _, _, c, first in jobs:
        assert torch.equal(c, first)
    x, graph = torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        _ck(lib.ane_op_gemm(ctypes.byref(jobs[0][0])))
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4 and torch.equal(jobs[0][3], jobs[0][4])


def test_fp32_products_give_their_memory_back_to_allocations():
    """An allocation that only fits with the block for the parts succeeds, and products go on without one (in a process of its own: for good)."""
    import os
    import subprocess
    import sys

    body = """
import numpy as np, torch
import test_gemm_gpu as t
rng = np.random.default_rng(5)
A, B = rng.standard_normal((1024, 768)).astype(np.float32), rng.standard_normal((768, 768)).astype(np.float32)
want = A.astype(np.float64) @ B.astype(np.float64).T
run = lambda: t._gemm(t.ane.DTYPE_F32, A, B, np.zeros((1024, 768), np.float32), 1024, 768, 768, 0, 0, 1)
first = run()
room = [t.lib.ane_dev_malloc(32 << 20) for _ in range(2)]
filler = t.lib.ane_dev_malloc(torch.cuda.mem_get_info()[0] + (32 << 20))
assert filler
for p in room:
    t.lib.ane_dev_free(p)
second = run()
assert t.rel_l2(first, want) < 2e-7 and t.rel_l2(second, want) < 1e-6 and (first != second).any()
t.lib.ane_dev_free(filler)
"""
    here = os.path.dirname(os.path.abspath(__file__))
    path = os.pathsep.join([here, os.path.dirname(here), os.path.dirname(os.path.dirname(os.path.abspath(ane.__file__)))])
    r = subprocess.run([sys.executable, "-c", body], env=dict(os.environ, PYTHONPATH=path), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("M,N,K", [(8, 8, 200), (40, 136, 72), (72, 24, 1000), (200, 8, 64), (264, 328, 130)])
def test_split_precision_of_thin_operands(M, N, K):
    """MN-major operands of widths that are no multiple of a k-block, hi beside lo: the tolerance of the other layouts above."""
    rng = np.random.default_rng(M + N)
    A, B, C0 = (rng.standard_normal(s).astype(np.float32) for s in ((K, M), (K, N), (M, N)))
    want = A.astype(np.float64).T @ B
    got = _gemm(ane.DTYPE_BF16X3, A, B, np.zeros((M, N), np.float32), M, N, K, 1, 1, 1)
    assert rel_l2(got, want) < 2e-5
    got = _gemm(ane.DTYPE_BF16X3, A, B, C0, M, N, K, 1, 1, 2)
    assert rel_l2(got, want + C0) < 2e-5


def test_split_precision_of_thin_operands_takes_little_memory():
    """A million rows of eight columns, twice: 64 MiB of halves and not 512.  Whole numbers: exact in any order of addition."""
    import torch
    rng = np.random.default_rng(7)
    K = 1 << 20
    A, B = (rng.integers(-1, 2, (K, 8)).astype(np.float32) for _ in range(2))
    filler = lib.ane_dev_malloc(torch.cuda.mem_get_info()[0] - (300 << 20))
    assert filler
    try:
        got = _gemm(ane.DTYPE_BF16X3, A, B, np.zeros((8, 8), np.float32), 8, 8, K, 1, 1, 1)
    finally:
        lib.ane_dev_free(filler)
    np.testing.assert_array_equal(got, A.T @ B)


def test_gemm_rejects_misaligned_pitch():
    A = np.zeros((16, 20), np.float32)  # 20 bf16 = 40 bytes per row: not a 16-byte multiple
    dA, dB, dC = _up_bf16(A), _up_bf16(A), _up(np.zeros((16, 16), np.float32))
    g = _ffi.GemmArgs()
    g.struct_size = ctypes.sizeof(_ffi.GemmArgs)
    g.dtype = ane.DTYPE_BF16
    g.d_a, g.d_b, g.d_c = dA, dB, dC
    g.m, g.n, g.k, g.lda, g.ldb, g.ldc, g.out_mode, g.alpha = 16, 16, 20, 20, 20, 16, 1, 1.0
    assert lib.ane_op_gemm(ctypes.byref(g)) != 0
    assert b"16-byte" in lib.ane_ops_last_error()
    for p in (dA, dB, dC):
        lib.ane_dev_free(p)


def _gradients_in_a_child(env, cases):
    """Gradients of one micro-step by tensor for each case, from a process with `env`."""
    import os
    import subprocess
    import sys
    import tempfile
    code = """
import sys
import numpy as np
import ane
out = {}
for i, (dim, hidden, heads, layers, vocab, seq, batch, arch, dtype) in enumerate(%r):
    rng = np.random.default_rng(7)
    e = ane.open(ane.Options(dim=dim, hidden=hidden, n_layers=layers, n_heads=heads, n_kv_heads=heads, vocab=vocab, seq=seq, batch=batch, seed=3,
                             arch=arch, quirks=0, compute_dtype=dtype, accum_steps=1000))
    for tid in (ane.T_WQ, ane.T_WK, ane.T_WV, ane.T_WO, ane.T_W1, ane.T_W2, ane.T_W3):
        for l in range(layers):
            n = e.tensor_size(tid, l)
            if n > 0:
                e.import_tensor(tid, l, (0.05 * rng.standard_normal(n)).astype(np.float32))
    e.import_tensor(ane.T_EMBED, 0, (0.05 * rng.standard_normal(e.tensor_size(ane.T_EMBED, 0))).astype(np.float32))
    tokens = rng.integers(0, vocab, (batch, seq + 1)).astype(np.uint16)
    assert e.step_tokens(tokens[:, :-1].copy(), tokens[:, 1:].copy()).device_status == 0
    for tid in (ane.T_EMBED, ane.T_WQ, ane.T_WO, ane.T_W1, ane.T_W2):
        out["%%d %%d" %% (i, tid)] = e.export_tensor(tid, 0, ane.engine.G)
    e.close()
np.savez(sys.argv[1], **out)
""" % (cases,)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "autoresearch-go-ane_b200"), **env)
    with tempfile.TemporaryDirectory() as where:
        path = os.path.join(where, "g.npz")
        done = subprocess.run([sys.executable, "-c", code, path], env=env, capture_output=True, text=True, timeout=300)
        assert done.returncode == 0, done.stderr[-2000:]
        return dict(np.load(path))


def test_products_in_shares_behind_a_norm():
    """Gradients with the dX products of few tiles shared out along the contraction (their sums added by the norm's backward)
    against whole ones.  At split precision what differs is the order of fp32 sums: K / 16 additions, each off by up to 2^-24 of
    the sum, 9e-6 at K = 2304; 2e-5 for what three layers of it amount to.  In bf16 a difference d of a value moves its rounding
    (steps of u = 2^-8) with a probability of d / u, by u: sqrt(d u) in the mean, which three or four roundings on is the roundings' own
    size.  So both are two chains of independent roundings, some 18 of 1.6e-3 in three layers: sqrt(2 * 18) * 1.6e-3 = 1e-2; a share
    that is left out or added twice is off by tenths.  Rows that end inside a tile, fewer rows than a tile, a contraction with a
    remainder, no weights of the norm (reference architecture)."""
    cases = [
        (288, 768, 6, 3, 1000, 100, 1, ane.ARCH_LLAMA, ane.DTYPE_BF16),
        (768, 2048, 12, 2, 4096, 256, 1, ane.ARCH_LLAMA, ane.DTYPE_BF16),
        (200, 544, 5, 3, 504, 67, 3, ane.ARCH_LLAMA, ane.DTYPE_BF16),
        (128, 512, 2, 3, 2000, 128, 3, ane.ARCH_REFERENCE, ane.DTYPE_BF16),
        (320, 768, 5, 3, 1000, 300, 1, ane.ARCH_REFERENCE, ane.DTYPE_BF16X3),
    ]
    whole, shares = _gradients_in_a_child({"ANE_B200_GEMM_PARTS": "0"}, cases), _gradients_in_a_child({}, cases)
    assert whole.keys() == shares.keys()
    for i, case in enumerate(cases):
        differ = 0
        for key in [k for k in whole if k.startswith(f"{i} ")]:
            a, b = whole[key].astype(np.float64), shares[key].astype(np.float64)
            assert np.isfinite(b).all() and np.linalg.norm(a) > 0
            off = np.linalg.norm(a - b) / np.linalg.norm(a)
            differ += off > 0
            assert off < (2e-5 if case[-1] == ane.DTYPE_BF16X3 else 1e-2), (case, key, off)
        assert differ > 0, case  # the sums were formed in another order
