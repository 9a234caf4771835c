"""The grouped product of a portion of few slots (17 to 511), bf16: through the slot list, without a workspace, as exact as multiply-adds."""
import math
import os
import subprocess
import sys

import numpy as np
import pytest

from device_util import BF16, as_dt, dev, from_dt, i32, release, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


class Portion:
    def __init__(self, G, T, top, E, N, K, identity=0, seed=1):
        r = np.random.default_rng(seed)
        self.G, self.lib, self.T, self.top, self.E, self.N, self.K, self.identity = G, G.cuda_lib(), T, top, E, N, K, identity
        self.idx = i32(np.stack([r.permutation(E)[:top] for _ in range(T)])) if top <= E else i32(r.integers(0, E, (T, top)))
        (self.wf, w), (self.af, a) = as_dt(BF16, r.standard_normal((E - identity, N, K))), as_dt(BF16, r.standard_normal((T, K)))
        self.w, self.a = dev(G, w), dev(G, a)
        self.ws = zeros(G, 4 * self.lib.ggb_moe_group_ints(T * top, E))
        self.c = zeros(G, T * top * N * 4)
        G.check(self.lib.ggb_op_moe_group_identity(dev(G, self.idx).ptr, T, top, E, identity, self.ws.ptr))
        G.sync()

    def launch(self, act=0, a=None, w=None, c=None, ldc=None, gather=1):
        return self.lib.ggb_op_moe_linear_identity(BF16, w or self.w.ptr, self.N, self.K, a or self.a.ptr, self.K, gather, self.T, self.top, self.E, self.identity, self.ws.ptr,
                                                   act, 0.0, 0.0, c or self.c.ptr, ldc or self.N)

    def rows(self):
        """(expert, token) of every row of the product"""
        n = self.T * self.top
        lists = self.ws.download(np.int32)[self.E + 1:]
        row_src, row_expert = lists[:n], lists[2 * n + 2 * self.lib.ggb_moe_max_tiles(n, self.E) + 1:][:n]
        return row_expert, row_src

    def want(self):
        e, t = self.rows()
        real = e < self.E - self.identity
        return real, np.einsum("rnk,rk->rn", self.wf[e[real]], self.af[t[real]])


@pytest.mark.parametrize("T,top,E,N,K,identity", [(5, 4, 8, 96, 192, 0), (17, 1, 1, 32, 256, 0), (70, 1, 2, 160, 1024, 0), (65, 1, 1, 128, 192, 0), (127, 4, 32, 96, 320, 0),
                                                  (30, 3, 40, 64, 192, 8), (9, 2, 300, 32, 640, 0)])
def test_through_the_slot_list(gpu, T, top, E, N, K, identity):
    p = Portion(gpu, T, top, E, N, K, identity)
    gpu.check(p.launch())
    real, want = p.want()
    got = p.c.download(np.float32).reshape(T * top, N)
    # exact products; a block of 64 is summed by the tensor cores (its largest partial sum, truncated to 2^-23 of it at each of 4 steps), the blocks in fp32
    assert np.abs(got[real] - want).max() < (4 * 2.0 ** -23 * 8 * 8 + K / 64 * 2.0 ** -24 * 6) * np.sqrt(K)
    assert not got[~real].any()
    # rows in slot order already, activation, a longer row of results
    e, t = p.rows()
    _, rows = as_dt(BF16, p.af[t])
    y = zeros(gpu, T * top * (N + 8) * 2)
    gpu.check(p.launch(act=4, a=dev(gpu, rows).ptr, c=y.ptr, ldc=N + 8, gather=0))
    act = from_dt(BF16, y, (T * top, N + 8))
    z = got[real].astype(np.float64)
    gelu = 0.5 * z * (1 + np.vectorize(math.erf)(z / math.sqrt(2)))
    assert np.abs(act[real][:, :N] - gelu).max() <= 2.0 ** -8 * np.abs(gelu).max() and not act[:, N:].any()


@pytest.mark.parametrize("K", [64, 128, 256, 2048, 8192])
def test_error_is_no_larger_than_that_of_multiply_adds(gpu, K):
    p = Portion(gpu, 20, 2, 2, 256, K)
    gpu.check(p.launch())
    real, want = p.want()
    e, t = p.rows()
    chain = np.zeros(want.shape)
    for k in range(K):  # fmaf in k order: the products of bf16 numbers are exact, one rounding a step
        chain = (chain + p.wf[e, :, k] * p.af[t, k][:, None]).astype(np.float32).astype(np.float64)
    err = lambda x: np.linalg.norm(x - want) / np.linalg.norm(want)  # noqa: E731
    assert err(p.c.download(np.float32).reshape(want.shape)) <= err(chain) * 1.001  # (equal sums where the tile kernel takes them)


def test_a_matrix_and_results_off_their_boundaries(gpu):
    """A matrix that starts between two 16-byte pieces, results between two 8-byte ones: any address of the type is taken."""
    p = Portion(gpu, 6, 4, 4, 64, 192)
    gpu.check(p.launch())
    want = p.c.download(np.float32).reshape(24, 64)
    w = zeros(gpu, 4 * 64 * 192 * 2 + 2)
    _, raw = as_dt(BF16, p.wf)
    w.upload(np.concatenate([np.zeros(1, np.uint16), raw.reshape(-1).view(np.uint16)]))
    gpu.check(p.launch(w=w.ptr.value + 2))
    assert np.abs(p.c.download(np.float32).reshape(24, 64) - want).max() < 2e-4
    y = zeros(gpu, 24 * 64 * 2 + 2)
    gpu.check(p.launch(act=1, c=y.ptr.value + 2))
    got = (y.download(np.uint16)[1:1 + 24 * 64].astype(np.uint32) << 16).view(np.float32).reshape(24, 64)
    relu2 = np.square(np.maximum(want.astype(np.float64), 0))
    assert np.abs(got - relu2).max() <= 2.0 ** -8 * relu2.max()


CAPTURE = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np
import gemma_ggml_b200 as G
from test_moe_few_slots_gpu import Portion

G.init(0)
lib, p, big = G.cuda_lib(), Portion(G, 8, 4, 8, 64, 256), Portion(G, 2048, 4, 8, 64, 256, seed=2)
G.check(lib.ggb_capture_begin())
rc = p.launch()
g = C.c_void_p()
G.check(lib.ggb_capture_end(C.byref(g)))
G.check(rc, "captured product")
G.check(lib.ggb_graph_launch(g))
real, want = p.want()
def close():
    return np.abs(p.c.download(np.float32).reshape(want.shape) - want).max() < 1e-3
assert close()
G.check(big.launch())  # takes a workspace of 8192 rows
G.sync()
p.c.zero()
G.check(lib.ggb_graph_launch(g))
assert close()
assert np.abs(big.c.download(np.float32).reshape(8192, 64) - big.want()[1]).max() < 1e-3
print("ok")
"""


def test_a_first_product_inside_a_capture_and_a_larger_one_behind_it():
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", CAPTURE, os.path.dirname(tests), tests], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
