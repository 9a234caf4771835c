"""The quantised GEMM of the prefill (csrc/prefill.cu) at the edges of its tiles: one CTA of 128 rows, pairs of CTAs of 256 and 512, columns of
64 to 256, pieces of K in tensor memory and over CTAs; gate | up with gelu(gate) * up behind it.  Against a float64 product of the same
bf16 operands: products are exact, the tensor cores truncate a running sum by at most 2^-23 of it once per 16 of K."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O
from device_util import dev, f32, release, zeros
from safolorn_fixture import bf16_round

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def matrix(gpu, r, wtype, N, K):
    q = O.quantize(wtype, f32(r.standard_normal((N, K)) * 0.02))
    return gpu.Weight.upload(wtype, q, K), bf16_round(O.dequantize(wtype, q, K))[0]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("wtype", [O.TYPE_Q4_0, O.TYPE_Q8_0])
@pytest.mark.parametrize("T,N,K,resid", [(1, 32, 64, 0), (128, 96, 576, 1), (129, 32, 64, 0), (200, 288, 128, 1), (256, 2080, 192, 0), (257, 64, 1024, 1), (512, 256, 2048, 1), (513, 544, 320, 0),
                                         (130, 4096, 64, 0), (300, 2048, 4096, 1), (70, 1056, 2112, 1),
                                         # pairs of 512 rows x 64, 64 (two accumulators), 128 and 256 columns
                                         (898, 2368, 64, 1), (795, 2368, 640, 0), (826, 4736, 64, 0), (277, 9536, 64, 1),
                                         # pairs of 256 rows: 64 x 8 accumulators, 128 x 4, 256 x 2, 256 x 2 x 4 CTAs along K, 128 x 8 CTAs
                                         (270, 800, 2048, 0), (297, 2464, 1024, 1), (130, 10176, 512, 0), (276, 1184, 3200, 1), (282, 288, 2240, 0)])
def test_products(gpu, wtype, T, N, K, resid):
    r = np.random.default_rng(T + N + K)
    w, wv = matrix(gpu, r, wtype, N, K)
    av, ar = bf16_round(r.standard_normal((T, K)))
    x = f32(r.standard_normal((T, N)))
    lib = gpu.cuda_lib()
    n_ws = lib.ggb_gemm_workspace_bytes(T, N, K)
    a, c, dx = dev(gpu, ar), zeros(gpu, T * N * 4), dev(gpu, x)
    for ws in (zeros(gpu, n_ws), None):
        gpu.check(lib.ggb_op_gemm_bf16(w.h, a.ptr, T, c.ptr, N, dx.ptr if resid else None, ws.ptr if ws else None, n_ws if ws else 0))
        want = av @ wv.T + (x if resid else 0.0)
        assert rel(c.download(np.float32).reshape(T, N), want) < (K / 16 + 8) * 2.0 ** -23 + 1e-7


@pytest.mark.parametrize("wtype", [O.TYPE_Q4_0, O.TYPE_Q8_0])
@pytest.mark.parametrize("T,N,K", [(257, 512, 2048), (300, 2048, 4096), (276, 1184, 3200), (129, 512, 2048), (70, 1056, 2112), (270, 800, 2048)])
def test_pieces_of_k_are_added_in_order(gpu, wtype, T, N, K):
    """With a workspace, a product is the sum of its pieces along K, the first to the last, whether one CTA or several summed them."""
    r, lib = np.random.default_rng(K), gpu.cuda_lib()
    q, ar = O.quantize(wtype, f32(r.standard_normal((N, K)) * 0.02)), bf16_round(r.standard_normal((T, K)))[1]
    n_ws, x, c = lib.ggb_gemm_workspace_bytes(T, N, K), f32(r.standard_normal((T, N))), zeros(gpu, T * N * 4)
    w, pieces = gpu.Weight.upload(wtype, q, K), lib.ggb_gemm_pieces(T, N, K)
    assert pieces > 1
    gpu.check(lib.ggb_op_gemm_bf16(w.h, dev(gpu, ar).ptr, T, c.ptr, N, dev(gpu, x).ptr, zeros(gpu, n_ws).ptr, n_ws))
    step, want, y = -(-(K // 64) // pieces) * 64, None, zeros(gpu, T * N * 4)
    for k in range(0, K, step):
        n, row = min(step, K - k), q.shape[1] // (K // 32)
        part = gpu.Weight.upload(wtype, np.ascontiguousarray(q[:, k // 32 * row:(k + n) // 32 * row]), n)
        gpu.check(lib.ggb_op_gemm_bf16(part.h, dev(gpu, np.ascontiguousarray(ar[:, k:k + n])).ptr, T, y.ptr, N, None, None, 0))
        piece = y.download(np.float32).reshape(T, N)
        want = piece.copy() if want is None else want + piece
    assert (c.download(np.float32).reshape(T, N) == want + x).all()


@pytest.mark.parametrize("T,N,K", [(128, 96, 576), (300, 2048, 4096), (257, 64, 1024), (512, 256, 2048), (129, 32, 64)])
def test_outputs_that_start_anywhere(gpu, T, N, K):
    """Results and residuals on any 4-byte boundary, whether the product is cut along K in tensor memory, over CTAs or not at all."""
    r = np.random.default_rng(T)
    w, _ = matrix(gpu, r, O.TYPE_Q8_0, N, K)
    lib, a, x = gpu.cuda_lib(), dev(gpu, bf16_round(r.standard_normal((T, K)))[1]), f32(r.standard_normal((T, N)))
    n_ws = lib.ggb_gemm_workspace_bytes(T, N, K)
    ws, got = zeros(gpu, n_ws), []
    for skip in (0, 1, 2, 3):
        c, dx = zeros(gpu, (T * N + 8) * 4), dev(gpu, np.concatenate([np.zeros(skip, np.float32), x.reshape(-1)]))
        for with_ws in (True, False):
            gpu.check(lib.ggb_op_gemm_bf16(w.h, a.ptr, T, c.ptr.value + 4 * skip, N, dx.ptr.value + 4 * skip, ws.ptr if with_ws else None, n_ws if with_ws else 0))
            y = c.download(np.float32)
            assert not y[:skip].any() and not y[skip + T * N:].any()
            got.append(y[skip:skip + T * N])
    for i in range(2, 8):
        assert (got[i] == got[i % 2]).all()


@pytest.mark.parametrize("wtype", [O.TYPE_Q4_0, O.TYPE_Q8_0])
@pytest.mark.parametrize("T,F,K", [(129, 256, 64), (300, 512, 320), (512, 1024, 256), (700, 256, 1024), (270, 5120, 64), (600, 5120, 192)])  # the last two: pairs of 512 rows
def test_gate_up_gelu(gpu, wtype, T, F, K):
    r = np.random.default_rng(T + F)
    (g, gv), (u, uv) = matrix(gpu, r, wtype, F, K), matrix(gpu, r, wtype, F, K)
    av, ar = bf16_round(4.0 * r.standard_normal((T, K)))
    lib = gpu.cuda_lib()
    a, y, y2 = dev(gpu, ar), zeros(gpu, T * F * 2), zeros(gpu, T * F * 2)
    gpu.check(lib.ggb_op_gemm_geglu_bf16(g.h, u.h, a.ptr, T, y.ptr))
    got = (y.download(np.uint16).astype(np.uint32) << 16).view(np.float32).reshape(T, F)
    z, up = av @ gv.T, av @ uv.T
    want = 0.5 * z * (1.0 + np.tanh(0.7978845608028654 * z * (1.0 + 0.044715 * z * z))) * up
    assert rel(got, want) < 3e-3  # gate and gelu rounded to fp16 (2^-11 each), the product to bf16 (2^-9)
    # the two launches it stands for
    cg, cu = zeros(gpu, T * F * 4), zeros(gpu, T * F * 4)
    gpu.check(lib.ggb_op_gemm_bf16_multi(2, (C.c_void_p * 2)(g.h, u.h), a.ptr, T, (C.c_void_p * 2)(cg.ptr, cu.ptr), (C.c_int64 * 2)(F, F), None, 0))
    gpu.check(lib.ggb_op_geglu_bf16(cg.ptr, cu.ptr, T * F, y2.ptr))
    assert (y.download(np.uint16) == y2.download(np.uint16)).all()  # the same sums, the same table
    assert lib.ggb_op_gemm_geglu_bf16(g.h, u.h, a.ptr, 128, y.ptr) != 0


def test_gelu_of_every_fp16_number(gpu):
    """One number of K: gate = code * d * a exactly, its fp16 number spread over all signs and exponents."""
    lib, T, F, K = gpu.cuda_lib(), 1024, 512, 64
    r = np.random.default_rng(5)
    w = f32(np.zeros((F, K)))
    w[:, 0] = r.integers(-127, 128, F)
    w[:, 1] = 127.0  # the block's scale is 1
    q = O.quantize(O.TYPE_Q8_0, w)
    g = gpu.Weight.upload(O.TYPE_Q8_0, q, K)
    u = gpu.Weight.upload(O.TYPE_Q8_0, O.quantize(O.TYPE_Q8_0, f32(np.ones((F, K)))), K)
    av = np.zeros((T, K))
    av[:, 0] = np.exp2(r.uniform(-24.0, 10.0, T)) * r.choice([-1.0, 1.0], T)
    av[:4, 0] = [0.0, np.inf, -np.inf, np.nan]
    a = dev(gpu, bf16_round(av)[1])
    y, y2, cg, cu = zeros(gpu, T * F * 2), zeros(gpu, T * F * 2), zeros(gpu, T * F * 4), zeros(gpu, T * F * 4)
    gpu.check(lib.ggb_op_gemm_geglu_bf16(g.h, u.h, a.ptr, T, y.ptr))
    gpu.check(lib.ggb_op_gemm_bf16_multi(2, (C.c_void_p * 2)(g.h, u.h), a.ptr, T, (C.c_void_p * 2)(cg.ptr, cu.ptr), (C.c_int64 * 2)(F, F), None, 0))
    gpu.check(lib.ggb_op_geglu_bf16(cg.ptr, cu.ptr, T * F, y2.ptr))
    assert len(np.unique(cg.download(np.float32).astype(np.float16).view(np.uint16))) > 20000
    assert (y.download(np.uint16) == y2.download(np.uint16)).all()


@pytest.mark.parametrize("heads,kv,ff,fused", [(8, 8, 1024, False), (2, 1, 1024, True)])
def test_narrow_gate_up_is_summed_in_pieces(gpu, heads, kv, ff, fused):
    """A gate | up no wider than the workspace of the other products is summed along K in as many pieces as they are: two launches."""
    m = gpu.GemmaModel(gpu.make_config(1024, 2, heads, kv, 256, ff, 2048, 256, wtype=gpu.TYPE_Q8_0))
    m.init_synthetic_weights()
    m.init_kv_cache()
    m.build_compute_graph()
    lib, T = gpu.cuda_lib(), 200
    assert lib.ggb_gemm_pieces(T, 2 * ff, 1024) > 1
    gpu.check(lib.ggb_prof_reset())
    gpu.check(lib.ggb_prof_enable(1))
    try:
        m.prefill(np.arange(T, dtype=np.int32))
    finally:
        gpu.check(lib.ggb_prof_enable(0))
    assert (gpu.prof_get("op_gelu")[1] == 0) == fused
    first = m.prefill_logits(T - 1).copy()
    m.prefill(np.arange(128, dtype=np.int32))  # buffers sized for the longer prompt
    m.prefill(np.arange(T, dtype=np.int32))
    assert (m.prefill_logits(T - 1) == first).all()
    m.close()
