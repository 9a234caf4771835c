"""What follows a product that is cut along K, in the kernel that adds its pieces (csrc/prefill.cu): the norm of the rows, and the rotation and storing of
q, k and v; the same bits as the launches that they stand for, whether the product is cut (with a workspace) or not."""
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


def weight(gpu, r, wtype, N, K):
    return gpu.Weight.upload(wtype, O.quantize(wtype, f32(r.standard_normal((N, K)) * 0.02)), K)


@pytest.mark.parametrize("T,N,K,resid", [(1, 32, 2048, 1), (9, 96, 576, 0), (70, 1056, 2112, 1), (130, 288, 2240, 0), (300, 2048, 4096, 1), (512, 2048, 2048, 1), (129, 64, 64, 1)])
def test_norm(gpu, T, N, K, resid):
    r, lib = np.random.default_rng(N + K), gpu.cuda_lib()
    w, a, nw = weight(gpu, r, O.TYPE_Q8_0, N, K), dev(gpu, bf16_round(r.standard_normal((T, K)))[1]), dev(gpu, f32(1.0 + 0.1 * r.standard_normal(N)))
    x, n_ws = dev(gpu, f32(r.standard_normal((T, N)))).ptr if resid else None, lib.ggb_gemm_workspace_bytes(T, N, K)
    c, y, c2, y2 = (zeros(gpu, T * N * b) for b in (4, 2, 4, 2))
    for ws, n in ((zeros(gpu, n_ws).ptr, n_ws), (None, 0)):
        gpu.check(lib.ggb_op_gemm_bf16(w.h, a.ptr, T, c.ptr, N, x, ws, n))
        gpu.check(lib.ggb_op_rms_norm_bf16(c.ptr, nw.ptr, 1e-6, N, T, y.ptr))
        gpu.check(lib.ggb_op_gemm_norm_bf16(w.h, a.ptr, T, c2.ptr, x, ws, n, nw.ptr, 1e-6, y2.ptr))
        assert (c.download(np.uint32) == c2.download(np.uint32)).all() and (y.download(np.uint16) == y2.download(np.uint16)).all()


@pytest.mark.parametrize("T,H,Hkv,d,K", [(1, 4, 1, 64, 2048), (17, 4, 4, 64, 2112), (130, 8, 1, 256, 2048), (300, 3, 1, 96, 576), (512, 8, 1, 256, 2048), (129, 2, 2, 32, 64)])
def test_rotation_and_cache(gpu, T, H, Hkv, d, K):
    r, lib = np.random.default_rng(T + H), gpu.cuda_lib()
    rows, ctx = (H * d, Hkv * d, Hkv * d), T + 5
    gpu.check(lib.ggb_rope_table_init(ctx, d, 10000.0))
    ws3 = [weight(gpu, r, O.TYPE_Q8_0, n, K) for n in rows]
    w, a = (C.c_void_p * 3)(*(x.h for x in ws3)), dev(gpu, bf16_round(r.standard_normal((T, K)))[1])
    pos = np.arange(3, 3 + T, dtype=np.int32)
    pos[-1] = ctx + 7  # past the table: its last row, as in the launch that this one stands for
    dp, n_ws = dev(gpu, pos), lib.ggb_gemm_workspace_bytes(T, sum((n + 255) // 256 * 256 for n in rows), K)
    for ws, n in ((zeros(gpu, n_ws).ptr, n_ws), (None, 0)):
        got = []
        for fused in (0, 1):
            o = [zeros(gpu, T * n_out * 4) for n_out in rows]
            c, kc, vc = (C.c_void_p * 3)(*(x.ptr for x in o)), zeros(gpu, ctx * Hkv * d * 2), zeros(gpu, ctx * Hkv * d * 2)
            if fused:
                gpu.check(lib.ggb_op_gemm_rope_store_bf16(w, a.ptr, T, c, ws, n, dp.ptr, H, Hkv, d, 0.125, kc.ptr, vc.ptr))
            else:
                gpu.check(lib.ggb_op_gemm_bf16_multi(3, w, a.ptr, T, c, (C.c_int64 * 3)(*rows), ws, n))
                gpu.check(lib.ggb_op_rope_kv_store_batch(*(x.ptr for x in o), dp.ptr, T, H, Hkv, d, 0.125, kc.ptr, vc.ptr))
            got.append((o[0].download(np.uint32), kc.download(np.uint16), vc.download(np.uint16)))
        for x, y in zip(*got):
            assert x.any() and (x == y).all()
