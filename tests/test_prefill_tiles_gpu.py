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
                                         (130, 4096, 64, 0), (300, 2048, 4096, 1), (70, 1056, 2112, 1)])
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
@pytest.mark.parametrize("T,F,K", [(129, 256, 64), (300, 512, 320), (512, 1024, 256), (700, 256, 1024)])
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
    assert np.mean(y.download(np.uint16) != y2.download(np.uint16)) < 1e-3  # the same sums; the table's gelu may round an fp16 number the other way
    assert lib.ggb_op_gemm_geglu_bf16(g.h, u.h, a.ptr, 128, y.ptr) != 0
