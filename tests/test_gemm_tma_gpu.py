"""Products of bf16 matrices (csrc/gemm.cu) against float64 at the edges of their tiles (rows of 128 and 256, columns of 64 to 256, pieces of
K) and of the groups of a mixture of experts.  Products are exact in fp32; the tensor cores truncate a running sum once per 16 of K, at most
2^-23 of it, so the error (2-norm) stays below K / 16 such steps of the result's norm."""
import numpy as np
import pytest

from device_util import BF16, as_dt, dev, from_dt, i32, release, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def limit(K):
    return (K / 16 + 8) * 2.0 ** -23 + 1e-7


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# what the rule of csrc/gemm.cu takes for them on 148 SMs: tiles of 128 rows
SINGLE = [(64, 32, 64, 0), (65, 96, 128, 4), (127, 256, 576, 0), (128, 288, 2112, 0), (129, 64, 4096, 0), (255, 2048, 2048, 8), (256, 2080, 192, 0), (257, 544, 1024, 0),
          (300, 4096, 64, 0), (1000, 1056, 1408, 0), (1024, 8192, 256, 0), (64, 160, 8192, 0), (2048, 32, 320, 0), (700, 8224, 448, 0),
          (528, 3744, 512, 0), (142, 5184, 1024, 0), (155, 9760, 512, 4), (650, 9600, 192, 0), (67, 2432, 4928, 0)]
# two CTAs a tile of 256 x 256: accumulators a CTA x CTAs along K 2 x 1, 1 x 8 (two rounds of tiles), 2 x 2, 2 x 4, and 1 x 1 in several rounds
PAIRS = [(131, 10368, 960, 0), (141, 2528, 5184, 8), (154, 5280, 5184, 0), (260, 1568, 5824, 0), (385, 9952, 704, 0), (1024, 8192, 2048, 0)]


@pytest.mark.parametrize("T,N,K,pad", SINGLE + PAIRS)
def test_dense(gpu, T, N, K, pad):
    r = np.random.default_rng(T + N)
    (w, wr), (a, ar) = as_dt(BF16, r.standard_normal((N, K))), as_dt(BF16, r.standard_normal((T, K)))
    dw, da, c, y = dev(gpu, wr), dev(gpu, ar), zeros(gpu, T * (N + pad) * 4), zeros(gpu, T * N * 2)
    lib = gpu.cuda_lib()
    gpu.check(lib.ggb_op_linear(BF16, dw.ptr, N, K, da.ptr, K, T, c.ptr, N + pad), "linear")
    want = a @ w.T
    got = c.download(np.float32).reshape(T, N + pad).astype(np.float64)
    assert rel(got[:, :N], want) < limit(K) and not got[:, N:].any()
    gpu.check(lib.ggb_op_linear_act(BF16, dw.ptr, N, K, da.ptr, K, T, 1, y.ptr), "linear_act")
    assert rel(from_dt(BF16, y, (T, N)), np.maximum(want, 0) ** 2) < 2.5e-3


@pytest.mark.parametrize("E,top,T,N,K", [(8, 2, 256, 96, 64), (3, 3, 200, 288, 192), (32, 4, 333, 1408, 256), (300, 2, 260, 32, 64), (5, 1, 777, 64, 128), (2, 1, 520, 320, 1024)])
def test_grouped(gpu, E, top, T, N, K):
    r = np.random.default_rng(E + T)
    lib = gpu.cuda_lib()
    (w, wr), (a, ar) = as_dt(BF16, r.standard_normal((E, N, K))), as_dt(BF16, r.standard_normal((T, K)))
    p = r.random(E) ** 4 + 1e-9  # a few experts take most rows, some none
    idx = np.stack([r.choice(E, top, replace=False, p=p / p.sum()) for _ in range(T)]) if top < E else np.tile(np.arange(E), (T, 1))
    ws, c = zeros(gpu, 4 * lib.ggb_moe_group_ints(T * top, E)), zeros(gpu, T * top * N * 4)
    gpu.check(lib.ggb_op_moe_group(dev(gpu, i32(idx)).ptr, T, top, E, ws.ptr), "group")
    gpu.check(lib.ggb_op_moe_linear(BF16, dev(gpu, wr).ptr, N, K, dev(gpu, ar).ptr, K, 1, T, top, E, ws.ptr, 0, c.ptr, N), "moe_linear")
    inv = ws.download(np.int32)[E + 1 + T * top:E + 1 + 2 * T * top].reshape(T, top)
    got = c.download(np.float32).reshape(T * top, N).astype(np.float64)[inv]
    want = np.empty((T, top, N))
    for e in range(E):
        t, s = np.nonzero(idx == e)
        want[t, s] = a[t] @ w[e].T
    assert rel(got, want) < limit(K)
