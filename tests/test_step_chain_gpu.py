"""Chains of short kernels of few tokens, each launched before the one ahead of it has ended: buffers written in turn, so that a kernel that
reads early meets old numbers and one that writes early destroys what is still read.  The same bits with a synchronisation behind each, without
one, and replayed as a graph."""
import ctypes as C

import numpy as np
import pytest

from device_util import BF16, F32, as_dt, at, dev, f32, i32, release, size_of, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


@pytest.mark.parametrize("dt,W,T", [(BF16, 2048, 1), (BF16, 200, 8), (BF16, 129, 3), (F32, 512, 1), (F32, 37, 5)])
def test_chain(gpu, dt, W, T):
    r = np.random.default_rng(W)
    lib, links = gpu.cuda_lib(), 12
    w, _ = as_dt(dt, r.standard_normal((links, W, W)) * (1.2 / W) ** 0.5)
    ws = [dev(gpu, as_dt(dt, w[i])[1]) for i in range(links)]
    x0 = as_dt(dt, r.standard_normal((T, W)))[1]
    bufs = [dev(gpu, x0), zeros(gpu, x0.nbytes)]

    def chain(sync):
        for i in range(links):
            gpu.check(lib.ggb_op_linear_act(dt, ws[i].ptr, W, W, bufs[i % 2].ptr, W, T, 4, bufs[(i + 1) % 2].ptr), "linear_act")
            if sync:
                gpu.sync()

    def start():
        bufs[0].upload(x0)
        gpu.sync()

    start()
    chain(True)
    want = bufs[0].download(x0.dtype)
    assert want.any()
    for _ in range(20):
        start()
        chain(False)
        assert (bufs[0].download(x0.dtype) == want).all()
    start()
    gpu.check(lib.ggb_capture_begin(), "capture_begin")
    chain(False)
    g = C.c_void_p()
    gpu.check(lib.ggb_capture_end(C.byref(g)), "capture_end")
    for _ in range(20):
        start()
        gpu.check(lib.ggb_graph_launch(g), "graph_launch")
        assert (bufs[0].download(x0.dtype) == want).all()
    gpu.check(lib.ggb_graph_free(g), "graph_free")


class Sublayers:
    """Calls that read and write a stream x of fp32 rows through a normed copy h, as a layer's sublayers do."""

    def __init__(self, gpu, dt, T, W, seed):
        self.gpu, self.lib, self.dt, self.T, self.W, self.r, self.calls = gpu, gpu.cuda_lib(), dt, T, W, np.random.default_rng(seed), []
        self.x0 = f32(self.r.standard_normal((T, W)))
        self.x, self.h, self.y = dev(gpu, self.x0), zeros(gpu, T * W * size_of(dt)), zeros(gpu, T * W * 4)
        self.pos, self.table = dev(gpu, i32([100])), dev(gpu, i32([3, 0, 2, 1]))

    def call(self, name, *args):
        args = [a.ptr if hasattr(a, "ptr") else a for a in args]
        self.calls.append((name, args))

    def mat(self, *shape):
        return dev(self.gpu, as_dt(self.dt, self.r.standard_normal(shape) * shape[-1] ** -0.5)[1])

    def vec(self, *shape, lo=0.5, hi=1.5):
        return dev(self.gpu, f32(self.r.uniform(lo, hi, shape)))

    def buf(self, n, size=4):
        return zeros(self.gpu, n * size)

    def norm(self, y):  # x += y, h = norm(x)
        none = (None, None, None, 0, 0, 0, None, None, 0, None, None, None)
        self.call("ggb_op_residual_layer_norm", self.dt, self.x, y, *none, self.vec(self.W), self.vec(self.W), 1e-5, self.W, self.T, None, self.x, self.h)

    def linear(self, a, N, K, c):
        self.call("ggb_op_linear", self.dt, self.mat(N, K), N, K, a, K, self.T, c, N)

    def go(self, rounds, sync):
        for _ in range(rounds):
            for name, args in self.calls:
                self.gpu.check(getattr(self.lib, name)(*args), name)
                if sync:
                    self.gpu.sync()

    def result(self):
        return self.x.download(np.float32)


def attention_sublayer(s, kind):
    T, W, H, G, D, dt = s.T, s.W, 4, 2, 64, s.dt
    N, HD, cos_sin = (H + 2 * G) * D, H * D, s.vec(256, D // 2, 2, lo=-1.0, hi=1.0)
    pr, q, o = s.buf(T * N), s.buf(T * HD), s.buf(T * HD, size_of(dt))
    cache = dev(s.gpu, as_dt(dt, s.r.standard_normal((256, int(s.lib.ggb_window_cache_ld(G, D, D)))))[1])
    s.linear(s.h, N, W, pr)
    k, v = at(pr, 4 * HD), at(pr, 4 * (HD + G * D))
    if kind == "sigmoid":
        s.call("ggb_op_sigmoid_qkv_store", dt, pr, k, v, N, T, H, G, D, D, 0.1, 64, 1e-5, D ** -0.5, s.pos, s.table, 64, cache, q)
        s.call("ggb_op_sigmoid_attn", dt, q, cache, s.table, 64, s.pos, T, H, G, D, D, 0, s.vec(H), s.vec(H), s.vec(H), o, s.buf(s.lib.ggb_sigmoid_attn_scratch_bytes(H), 1))
    else:
        s.call("ggb_op_head_qkv_store", dt, pr, k, v, N, T, H, G, D, D, s.vec(D), s.vec(D), 1e-5, D, 1, cos_sin, D ** -0.5, s.pos, s.table, 64, cache, q)
        s.call("ggb_op_masked_attn_gated", dt, q, cache, s.table, 64, s.pos, T, H, G, D, D, 0, 0, 30.0, None, None, 0, o, s.buf(s.lib.ggb_window_attn_scratch_bytes(H), 1))
    s.linear(o, W, HD, s.y)


def latent_sublayer(s):
    T, W, H, D, R, Dr, Dv, dt, ns = s.T, s.W, 4, 32, 128, 32, 32, s.dt, 3
    cos_sin = s.vec(256, Dr // 2, 2, lo=-1.0, hi=1.0)
    d, q, qa, o = s.buf(T * (R + Dr)), s.buf(T * H * (D + Dr)), s.buf(T * H * (R + Dr)), s.buf(T * H * Dv, size_of(dt))
    cache = dev(s.gpu, as_dt(dt, s.r.standard_normal((256, int(s.lib.ggb_latent_cache_ld(R, Dr)))))[1])
    part = s.buf(s.lib.ggb_latent_attn_scratch_bytes(T, H, R, ns), 1)
    s.linear(s.h, R + Dr, W, d)
    s.call("ggb_op_latent_kv_store", dt, d, R + Dr, T, R, Dr, Dr, s.vec(R), 1e-5, cos_sin, s.pos, s.table, 64, cache)
    s.linear(s.h, H * (D + Dr), W, q)
    s.call("ggb_op_latent_q_absorb", dt, q, H * (D + Dr), T, H, D, Dr, Dr, cos_sin, s.pos, s.mat(H, D, R), R, 0.1, qa)
    s.call("ggb_op_latent_attn", dt, qa, cache, s.table, 64, s.pos, T, H, R, Dr, ns, part)
    s.call("ggb_op_latent_attn_out", dt, part, ns, s.vec(H), s.mat(H, Dv, R), T, H, R, Dv, o)
    s.linear(o, W, H * Dv, s.y)


def experts_sublayer(s, kind):
    T, W, F, E, top, dt = s.T, s.W, 96, 8, 2, s.dt
    z, idx, wt, ws = s.buf(T * E), s.buf(T * top), s.buf(T * top), s.buf(s.lib.ggb_moe_group_ints(T * top, E))
    y1, y2, router = s.buf(T * top * F, size_of(dt)), s.buf(T * top * W), dev(s.gpu, f32(s.r.standard_normal((E, W)) * W ** -0.5))
    step = bool(s.lib.ggb_moe_step_form(T * top))
    if kind == "plain":
        s.call("ggb_op_moe_route", dt, s.h, W, T, router, s.vec(E), E, top, z, idx, wt)
        s.call("ggb_op_moe_group", idx, T, top, E, ws)
    else:
        if kind == "sigmoid":
            s.call("ggb_op_moe_route_sigmoid", dt, s.h, W, T, router, s.vec(E), E, top, 4, 2, z, idx, wt, ws if step else None)
        else:
            s.call("ggb_op_moe_route_softmax_groups", dt, s.h, W, T, router, s.vec(E), E, 0, top, 4, 2, 1.5, z, idx, wt, ws if step else None)
        if not step:
            s.call("ggb_op_moe_group", idx, T, top, E, ws)
    if kind == "softmax":  # an expert that every token uses, beside them
        up_s, a_s, c_s = s.mat(F, W), s.buf(T * F, size_of(dt)), s.buf(T * W)
        s.call("ggb_op_moe_linear_shared", dt, s.mat(E, F, W), F, W, s.h, W, 1, T, top, E, ws, 4, y1, F, up_s, F, W, s.h, W, a_s)
        s.call("ggb_op_moe_linear_shared", dt, s.mat(E, W, F), W, F, y1, F, 0, T, top, E, ws, 0, y2, W, s.mat(W, F), W, F, a_s, F, c_s)
        s.call("ggb_op_moe_combine", y2, ws, wt, T, top, E, W, s.y)
        s.norm(c_s)
    else:
        s.call("ggb_op_moe_linear", dt, s.mat(E, F, W), F, W, s.h, W, 1, T, top, E, ws, 4, y1, F)
        s.call("ggb_op_moe_linear", dt, s.mat(E, W, F), W, F, y1, F, 0, T, top, E, ws, 0, y2, W)
        s.call("ggb_op_moe_combine", y2, ws, wt, T, top, E, W, s.y)


SUBLAYERS = {"attention": lambda s: attention_sublayer(s, "soft"), "sigmoid attention": lambda s: attention_sublayer(s, "sigmoid"), "latent": latent_sublayer,
             "experts": lambda s: experts_sublayer(s, "plain"), "sigmoid router": lambda s: experts_sublayer(s, "sigmoid"), "soft-max router": lambda s: experts_sublayer(s, "softmax")}


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("T", [1, 3, 24])
@pytest.mark.parametrize("sub", list(SUBLAYERS))
def test_sublayers(gpu, sub, T, dt):
    s, rounds = Sublayers(gpu, dt, T, 256, T), 4
    s.norm(None)
    SUBLAYERS[sub](s)
    s.norm(s.y)

    def start():
        s.x.upload(s.x0)
        gpu.sync()

    start()
    s.go(rounds, True)
    want = s.result()
    assert np.isfinite(want).all() and (want != s.x0.reshape(-1)).any()
    for _ in range(10):
        start()
        s.go(rounds, False)
        assert (s.result() == want).all()
    start()
    gpu.check(s.lib.ggb_capture_begin(), "capture_begin")
    s.go(rounds, False)
    g = C.c_void_p()
    gpu.check(s.lib.ggb_capture_end(C.byref(g)), "capture_end")
    for _ in range(10):
        start()
        gpu.check(s.lib.ggb_graph_launch(g), "graph_launch")
        assert (s.result() == want).all()
    gpu.check(s.lib.ggb_graph_free(g), "graph_free")
