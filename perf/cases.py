"""Performance cases: the work that a user of this library has it do, through its public entry points.

A case is a plain dict; `kind` picks the entry point and the other fields are its sizes and options.  listed() names the ones that stand
for the ranges, draw() gives another one of the same ranges, prepare() makes what a program holds before the call, run() is one call (or the
few calls of one block), exact() the same result in 64 bits by plain torch.

Kinds
  offload    ggb_mul_mat with host pointers: the drop-in for the reference's mul_mat (Q4_0 / Q8_0 weights, Q8_0 rows)
  kquant     the packed K-quant mat-vec on an fp32 row (the mul_mat node of a q4_k_m model)
  decode     GemmaModel.decode_step: one token of a Q4_0 / Q8_0 Gemma model, and its logits
  prefill    GemmaModel.prefill: a prompt at once, and the logits of its last position
  linear     ggb_op_linear on plain bf16 / fp32 matrices
  experts    a mixture of experts: router, slot lists, both products, weighted sum
  layer      one step of a dense layer with gated attention (norm, projections, cache, attention, feed-forward), a captured graph as
             the engine replays it
  attention  ggb_op_masked_attn_gated / ggb_op_diff_attn over a paged cache: portions and steps
  sigmoid    ggb_op_sigmoid_attn over a paged cache
  latent     ggb_op_latent_attn and its output product over a paged latent cache
  delta      a portion of a recurrence: delta rule with a decay per head or per channel, lightning attention
"""
import ctypes as C
import math

import numpy as np
import torch

import gemma_ggml_b200 as G

BF16, F32 = G.TYPE_BF16, G.TYPE_F32
PAGE = 64  # positions per page of the paged cache, the engine's default
KIND_OF = {"bf16": (BF16, torch.bfloat16, 2), "f32": (F32, torch.float32, 4)}
Q_TYPE = {"q4_0": G.TYPE_Q4_0, "q8_0": G.TYPE_Q8_0, "q4_k": G.TYPE_Q4_K, "q6_k": G.TYPE_Q6_K}
Q_BYTES = {"q4_0": 18 / 32, "q8_0": 34 / 32, "q4_k": 144 / 256, "q6_k": 210 / 256}


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: the o projection of Gemma-2B as the reference's own program makes it, one token, host buffers
        dict(name="offload_q4_0_2048", kind="offload", q="q4_0", rows=2048, cols=2048, T=1),
        # one token through one dense layer of a bf16 model: eight short launches, latency more than bytes
        dict(name="layer_step_2048", kind="layer", dt="bf16", T=1, width=2048, heads=16, kv=4, dim=128, ff=8192, window=1024, pos=1800),
        # the output matrix of a q4_k_m Gemma-2B file (Q6_K, 256000 rows), once per token
        dict(name="kquant_logits_q6_k", kind="kquant", q="q6_k", rows=256000, cols=2048, T=1),
        # the headline: Gemma-2B Q4_0, batch-1 decode at 2048 positions
        dict(name="decode_2b_q4_0_2048", kind="decode", q="q4_0", embd=2048, layers=18, heads=8, kv=1, dim=256, ff=16384, vocab=256000, ctx=2048),
        # a feed-forward product of a prompt portion at the serving engine's portion size
        dict(name="linear_1024", kind="linear", dt="bf16", T=1024, N=8192, K=2048),
        # the float32 engine, a ragged portion
        dict(name="linear_f32_333", kind="linear", dt="f32", T=333, N=2816, K=1000),
        # a mixture-of-experts sublayer of a prompt portion
        dict(name="experts_1024", kind="experts", dt="bf16", T=1024, width=2048, ff=1408, experts=32, top=4),
        # soft-max attention of a prompt's second portion: window, kept first tokens, soft cap and gate
        dict(name="attention_1024", kind="attention", dt="bf16", maps=1, T=1024, pos=1024, heads=16, kv=4, dim=128, vdim=128, window=1024, keep=4, softcap=30.0, gate=True),
        # unnormalised sigmoid attention with a distance penalty, a ragged portion
        dict(name="sigmoid_777", kind="sigmoid", dt="bf16", T=777, pos=1024, heads=16, kv=4, dim=128, vdim=128, window=0),
        # latent attention, absorbed form, a prompt's second portion
        dict(name="latent_1024", kind="latent", dt="bf16", T=1024, pos=1024, heads=16, rank=512, rot=64, vdim=128, window=0),
        # the recurrence of a prompt portion, fp32 state
        dict(name="delta_1024", kind="delta", rule="head", T=1024, heads=16, kv=8, dim=128, vdim=128),
        # the largest: a 512-token prompt through Gemma-2B Q8_0
        dict(name="prefill_2b_q8_0_512", kind="prefill", q="q8_0", embd=2048, layers=18, heads=8, kv=1, dim=256, ff=16384, vocab=256000, T=512),
    ]


def draw(rng):
    def size(lo, hi, step=1):
        """a multiple of `step` in [lo, hi], even over the logarithm"""
        return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))) / step)) * step)

    def tokens(hi):
        return rng.choice([1, 1, size(2, 31), size(32, hi), size(32, hi), size(32, hi)])

    kind = rng.choice(["offload", "layer", "kquant", "decode", "linear", "linear", "experts", "attention", "attention", "sigmoid", "latent", "delta", "prefill"])
    dt = rng.choice(["bf16", "bf16", "bf16", "f32"])
    if kind == "offload":
        return dict(kind=kind, q=rng.choice(["q4_0", "q8_0"]), rows=size(64, 16384), cols=size(64, 8192, 32), T=rng.choice([1, 1, size(2, 8)]))
    if kind == "kquant":
        return dict(kind=kind, q=rng.choice(["q4_k", "q6_k"]), rows=size(256, 200000), cols=size(512, 4096, 256), T=1)
    if kind in ("decode", "prefill"):
        dim = rng.choice([64, 128, 256])
        heads = rng.choice([4, 8])
        c = dict(kind=kind, q=rng.choice(["q4_0", "q8_0"]), embd=size(512, 2048, 256), layers=rng.randint(2, 8), heads=heads, kv=rng.choice([1, heads]), dim=dim,
                 ff=size(1024, 8192, 512), vocab=size(4096, 64000, 256))
        return dict(c, ctx=size(64, 2048)) if kind == "decode" else dict(c, T=size(16, 512))
    if kind == "linear":
        whole = rng.random() < 0.75  # the sizes of models; the rest odd
        c = dict(kind=kind, dt=dt, T=tokens(2048), N=size(128, 12288, 64) if whole else size(65, 6000), K=size(128, 8192, 64) if whole else size(65, 3000))
        most = 4e9 if dt == "f32" or not whole else 1e11
        while 2.0 * c["T"] * c["N"] * c["K"] > most:
            c["T"] = max(1, c["T"] * 2 // 3)
        return c
    if kind == "experts":
        return dict(kind=kind, dt="bf16", T=tokens(1536), width=size(256, 2048, 64), ff=size(128, 2048, 64), experts=rng.choice([8, 16, 32]), top=rng.choice([2, 4]))
    if kind == "layer":
        dim, kv = rng.choice([64, 128]), rng.choice([1, 2, 4])
        return dict(kind=kind, dt=dt, T=rng.choice([1, 1, 1, size(2, 8)]), width=size(512, 4096, 64), heads=kv * rng.choice([1, 2, 4]), kv=kv, dim=dim,
                    ff=size(512, 8192, 64), window=rng.choice([0, 256, 1024]), pos=size(16, 2000))
    if kind in ("attention", "sigmoid"):
        kv, dim = rng.choice([1, 2, 4, 8]), rng.choice([64, 80, 96, 128])
        c = dict(kind=kind, dt=dt, T=tokens(1024), pos=rng.choice([0, size(1, 2000)]), heads=kv * rng.choice([1, 2, 4]), kv=kv, dim=dim, vdim=rng.choice([dim, 64, 128]),
                 window=rng.choice([0, 128, 512, 1024]))
        if kind == "sigmoid":
            return c
        maps = rng.choice([1, 1, 2])
        if maps == 2:
            c["dim"] = rng.choice([64, 128])
        return dict(c, maps=maps, keep=rng.choice([0, 4, 50]) if c["window"] else 0, softcap=rng.choice([0.0, 30.0]), gate=rng.random() < 0.5)
    if kind == "latent":
        return dict(kind=kind, dt=dt, T=tokens(1024), pos=rng.choice([0, size(1, 1500)]), heads=rng.choice([4, 8, 16]), rank=rng.choice([128, 256, 512]), rot=rng.choice([32, 64]),
                    vdim=rng.choice([64, 128]), window=rng.choice([0, 0, 512]))
    kv = rng.choice([2, 4, 8])
    return dict(kind="delta", rule=rng.choice(["head", "channel", "lightning"]), T=tokens(1024), heads=kv * rng.choice([1, 2]), kv=kv, dim=rng.choice([64, 96, 128]),
                vdim=rng.choice([64, 128]))


# ------------------------------------------------------------------------------------------------------------ inputs
class State:
    """What a program holds: the calls of one pass with their arguments bound, the outputs, and everything that must stay alive."""

    def __init__(self, **kw):
        self.calls, self.out, self.keep, self.graph, self.close = [], {}, [], None, None
        self.__dict__.update(kw)

    def ptr(self, t):
        if t is None:
            return C.c_void_p(None)
        self.keep.append(t)
        return C.c_void_p(t.data_ptr())

    def call(self, name, *args):
        fn = getattr(G.cuda_lib(), name)
        bound = [self.ptr(a) if a is None or isinstance(a, torch.Tensor) else a for a in args]
        self.calls.append((name, fn, [a if isinstance(a, C._SimpleCData) else t(a) for a, t in zip(bound, fn.argtypes)]))

    def __del__(self):
        try:
            G.sync()
            if self.graph is not None:
                G.cuda_lib().ggb_graph_free(self.graph)
            if self.close is not None:
                self.close()
        except Exception:
            pass


class Maker:
    def __init__(self, seed, device="cuda"):
        self.g = torch.Generator(device=device)
        self.g.manual_seed(int(seed) * 7919 + 12345)
        self.device = device

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(*shape, generator=self.g, device=self.device) * scale).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device=self.device) * (hi - lo) + lo

    def bytes(self, *shape):
        return torch.randint(0, 256, shape, generator=self.g, device=self.device, dtype=torch.uint8)

    def pages(self, n):
        """a page table: the pages of a sequence lie anywhere in the pool"""
        return torch.randperm(n, generator=self.g, device=self.device).to(torch.int32)


def rows_of(cache, table, n):
    """the first n positions of a paged cache, in order"""
    j = torch.arange(n, device=cache.device)
    return cache[table.long()[j // PAGE] * PAGE + j % PAGE]


def pos_dev(p):
    return torch.tensor([p, 0, 0, 0], dtype=torch.int32, device="cuda")


def attention_inputs(c, seed):
    m, maps = Maker(seed), c.get("maps", 1)
    _, tt, _ = KIND_OF[c["dt"]]
    n = c["pos"] + c["T"]
    pages = (n + PAGE - 1) // PAGE
    ld = (c["kv"] * (c["dim"] * maps + c["vdim"]) + 7) // 8 * 8
    d = dict(q=m.normal(c["T"], c["heads"], maps, c["dim"], scale=1.5 * c["dim"] ** -0.5), cache=m.normal(pages * PAGE, ld, dtype=tt), table=m.pages(pages))
    d["gate"] = m.normal(c["T"], c["heads"] * c["vdim"]) if c.get("gate") else None
    d["sink"] = m.normal(c["heads"]) if maps == 1 and not c.get("gate") else None  # the designs have a sink or a gate
    d["r1"], d["r2"], d["pb"] = m.uniform(0.2, 1.0, c["heads"]), m.uniform(0.1, 1.5, c["heads"]), m.uniform(-2.5, 0.0, c["heads"])
    return d


def latent_inputs(c, seed):
    m = Maker(seed)
    _, tt, _ = KIND_OF[c["dt"]]
    n, R, Dr, H = c["pos"] + c["T"], c["rank"], c["rot"], c["heads"]
    pages = (n + PAGE - 1) // PAGE
    ld = (R + Dr + 7) // 8 * 8
    return dict(qa=m.normal(c["T"], H, R + Dr, scale=1.5 * (R + Dr) ** -0.5), cache=m.normal(pages * PAGE, ld, dtype=tt), table=m.pages(pages), sink=m.normal(H),
                w_uv=m.normal(H * c["vdim"], R, scale=R ** -0.5, dtype=tt))


def linear_inputs(c, seed):
    m = Maker(seed)
    _, tt, _ = KIND_OF[c["dt"]]
    return dict(w=m.normal(c["N"], c["K"], scale=c["K"] ** -0.5, dtype=tt), a=m.normal(c["T"], c["K"], dtype=tt))


def experts_inputs(c, seed):
    m = Maker(seed)
    _, tt, _ = KIND_OF[c["dt"]]
    W, F, E = c["width"], c["ff"], c["experts"]
    return dict(h=m.normal(c["T"], W, dtype=tt), router=m.normal(E, W, scale=1.5 * W ** -0.5), bias=m.normal(E, scale=0.3), up=m.normal(E, F, W, scale=W ** -0.5, dtype=tt),
                down=m.normal(E, W, F, scale=F ** -0.5, dtype=tt))


def layer_inputs(c, seed):
    m = Maker(seed)
    _, tt, _ = KIND_OF[c["dt"]]
    T, W, H, Gk, D, F = c["T"], c["width"], c["heads"], c["kv"], c["dim"], c["ff"]
    n = c["pos"] + T
    pages = (n + PAGE - 1) // PAGE
    ld = (Gk * 2 * D + 7) // 8 * 8
    ang = torch.arange(n + 1, device="cuda", dtype=torch.float64)[:, None] * 10000.0 ** (-torch.arange(D // 2, device="cuda", dtype=torch.float64) * 2 / D)
    return dict(x=m.normal(T, W), nw=m.normal(2, W, scale=0.1) + 1.0, nb=m.normal(2, W, scale=0.1), proj=m.normal((2 * H + 2 * Gk) * D, W, scale=W ** -0.5, dtype=tt),
                qn=m.normal(D, scale=0.1) + 1.0, kn=m.normal(D, scale=0.1) + 1.0, cs=torch.stack([ang.cos(), ang.sin()], -1).float().contiguous(),
                cache=m.normal(pages * PAGE, ld, dtype=tt), table=m.pages(pages), o=m.normal(W, H * D, scale=(H * D) ** -0.5, dtype=tt),
                up=m.normal(F, W, scale=W ** -0.5, dtype=tt), down=m.normal(W, F, scale=F ** -0.5, dtype=tt))


def delta_inputs(c, seed):
    m = Maker(seed)
    T, H, Gk, D, Dv = c["T"], c["heads"], c["kv"], c["dim"], c["vdim"]
    if c["rule"] == "lightning":
        Gk = H
    ld = 2 * Gk * D + H * Dv
    x = m.normal(T, ld)
    if c["rule"] != "lightning":
        x = torch.nn.functional.silu(x)  # the projections come through a short convolution with silu
    return dict(x=x, Gk=Gk, ld=ld, b=m.normal(T, H), a=m.normal(T, H if c["rule"] == "head" else H * D), A_log=m.uniform(-1.0, 1.0, H),
                dt_bias=m.uniform(-4.0, 0.0, H if c["rule"] == "head" else H * D), decay=torch.exp(-1.0 / (2.0 * 2.0 ** (10.0 * torch.arange(H, device="cuda") / H))).float(),
                state=m.normal(H, D, Dv, scale=0.1))


def offload_inputs(c, seed):
    m = Maker(seed, "cpu")
    nb = c["cols"] // 32
    if c["q"] == "q4_0":
        w = m.bytes(c["rows"], nb, 18)
        w[:, :, 0:2] = m.uniform(0.002, 0.006, c["rows"], nb).half().view(torch.uint8).reshape(c["rows"], nb, 2)
    else:
        w = m.bytes(c["rows"], nb, 34)
        w[:, :, 0:2] = m.uniform(0.0002, 0.0006, c["rows"], nb).half().view(torch.uint8).reshape(c["rows"], nb, 2)
    a = m.bytes(c["T"], nb, 34)
    a[:, :, 0:2] = m.uniform(0.005, 0.03, c["T"], nb).half().view(torch.uint8).reshape(c["T"], nb, 2)
    return w.reshape(c["rows"], -1).numpy(), a.reshape(c["T"], -1).numpy()


def kquant_inputs(c, seed):
    m = Maker(seed)
    nb, size = c["cols"] // 256, 144 if c["q"] == "q4_k" else 210
    b = m.bytes(c["rows"], nb, size)
    d = m.uniform(0.0002, 0.0008, c["rows"], nb)
    if c["q"] == "q4_k":
        b[:, :, 0:2] = d.half().view(torch.uint8).reshape(c["rows"], nb, 2)
        b[:, :, 2:4] = (7.5 * d).half().view(torch.uint8).reshape(c["rows"], nb, 2)
    else:
        b[:, :, 208:210] = (d / 4).half().view(torch.uint8).reshape(c["rows"], nb, 2)
    return b.reshape(c["rows"], -1).contiguous(), m.normal(c["T"], c["cols"])


def gemma_config(c, seed):
    n_ctx = c["ctx"] if c["kind"] == "decode" else c["T"]
    return G.make_config(c["embd"], c["layers"], c["heads"], c["kv"], c["dim"], c["ff"], c["vocab"], n_ctx, wtype=Q_TYPE[c["q"]], seed=int(seed) % (1 << 30) + 1)


def prompt_of(c, seed):
    return np.random.default_rng(seed).integers(0, c["vocab"], size=1 if c["kind"] == "decode" else c["T"]).astype(np.int32)


# ------------------------------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    G.init(0)
    c, k = case, case["kind"]
    if k in ("decode", "prefill"):
        m = G.GemmaModel(gemma_config(c, seed))
        m.init_synthetic_weights()
        m.init_kv_cache()
        if k == "decode":
            m.fill_kv_cache_synthetic(seed)
        m.build_compute_graph()
        return State(kind=k, model=m, tokens=prompt_of(c, seed), pos=c.get("ctx", 0) - 1, close=m.close)
    if k == "offload":
        w, a = offload_inputs(c, seed)
        dst = np.zeros((c["T"], c["rows"]), dtype=np.float32)
        s = State(kind=k, w=w, a=a, dst=dst)
        s.args = (c["rows"], c["T"], 1, w.shape[1], c["T"], c["rows"] * 4, c["rows"] * 4 * c["T"], a.shape[1], c["cols"], w.ctypes.data_as(C.c_void_p),
                  dst.ctypes.data_as(C.c_void_p), Q_TYPE[c["q"]], a.ctypes.data_as(C.c_void_p))
        s.close = lambda: G.cuda_lib().ggb_mul_mat_forget(s_w)  # noqa: E731
        s_w = w.ctypes.data_as(C.c_void_p)
        G.check(G.cuda_lib().ggb_mul_mat(*s.args), "ggb_mul_mat")  # a program's weights have been used before
        return s
    s = State(kind=k)
    if k == "kquant":
        raw, x = kquant_inputs(c, seed)
        L, ty = G.cuda_lib(), Q_TYPE[c["q"]]
        pitch = raw.shape[1]
        packed = torch.empty(c["rows"] * pitch if c["q"] == "q4_k" else int(L.ggb_q6k_packed_bytes(c["rows"], c["cols"])), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        repack = L.ggb_op_q4k_repack if c["q"] == "q4_k" else L.ggb_op_q6k_repack
        G.check(repack(raw.data_ptr(), c["rows"], pitch, c["cols"], packed.data_ptr()), "repack")
        G.sync()
        s.out = dict(y=torch.empty(c["T"], c["rows"], device="cuda"))
        s.call("ggb_op_mul_mat_kq_packed_f32", ty, packed, c["rows"], c["cols"], x, c["T"], s.out["y"], c["rows"])
        return s
    if k == "delta":
        d = delta_inputs(c, seed)
        T, H, D, Dv, Gk, ld = c["T"], c["heads"], c["dim"], c["vdim"], d["Gk"], d["ld"]
        s.out = dict(o=torch.empty(T, H * Dv, device="cuda"), state=d["state"])
        s.keep.append(d["x"])
        base = d["x"].data_ptr()
        q, kk, v = (C.c_void_p(base + 4 * off) for off in (0, Gk * D, 2 * Gk * D))
        if c["rule"] == "head":
            s.call("ggb_op_gated_delta", q, kk, v, ld, d["b"], d["a"], H, T, H, Gk, D, Dv, d["A_log"], d["dt_bias"], d["state"], s.out["o"], H * Dv)
        elif c["rule"] == "channel":
            s.call("ggb_op_channel_delta", q, kk, v, ld, d["b"], H, d["a"], H * D, 0, T, H, Gk, D, Dv, d["A_log"], d["dt_bias"], d["state"], s.out["o"], H * Dv)
        else:
            s.call("ggb_op_lightning_attn", q, kk, v, ld, T, H, D, Dv, d["decay"], d["state"], s.out["o"], H * Dv)
        return s
    dt, tt, _ = KIND_OF[c["dt"]]
    T = c["T"]
    if k == "linear":
        d = linear_inputs(c, seed)
        s.out = dict(c=torch.empty(T, c["N"], device="cuda"))
        s.call("ggb_op_linear", dt, d["w"], c["N"], c["K"], d["a"], c["K"], T, s.out["c"], c["N"])
        return s
    if k == "experts":
        d = experts_inputs(c, seed)
        W, F, E, top = c["width"], c["ff"], c["experts"], c["top"]
        L = G.cuda_lib()
        z, idx, wt = torch.empty(T, E, device="cuda"), torch.empty(T, top, dtype=torch.int32, device="cuda"), torch.empty(T, top, device="cuda")
        ws = torch.zeros(int(L.ggb_moe_group_ints(T * top, E)), dtype=torch.int32, device="cuda")
        y1, y2 = torch.empty(T * top, F, dtype=tt, device="cuda"), torch.empty(T * top, W, device="cuda")
        s.out = dict(y=torch.empty(T, W, device="cuda"))
        s.call("ggb_op_moe_route", dt, d["h"], W, T, d["router"], d["bias"], E, top, z, idx, wt)
        s.call("ggb_op_moe_group", idx, T, top, E, ws)
        s.call("ggb_op_moe_linear", dt, d["up"], F, W, d["h"], W, 1, T, top, E, ws, 4, y1, F)  # 4: GGB_ACT_GELU_ERF
        s.call("ggb_op_moe_linear", dt, d["down"], W, F, y1, F, 0, T, top, E, ws, 0, y2, W)
        s.call("ggb_op_moe_combine", y2, ws, wt, T, top, E, W, s.out["y"])
        return s
    pos = pos_dev(c["pos"])
    if k == "layer":
        d = layer_inputs(c, seed)
        W, H, Gk, D, F = c["width"], c["heads"], c["kv"], c["dim"], c["ff"]
        N, HD, nil = (2 * H + 2 * Gk) * D, H * D, None
        L = G.cuda_lib()
        f32 = lambda *shape: torch.empty(*shape, device="cuda")  # noqa: E731
        h, pr, qr, ya, yf = torch.empty(T, W, dtype=tt, device="cuda"), f32(T, N), f32(T, HD), f32(T, W), f32(T, W)
        ao, act = torch.empty(T, HD, dtype=tt, device="cuda"), torch.empty(T, F, dtype=tt, device="cuda")
        h2, scratch = torch.empty(T, W, dtype=tt, device="cuda"), torch.empty(int(L.ggb_window_attn_scratch_bytes(H)), dtype=torch.uint8, device="cuda")
        x1, x2 = f32(T, W), f32(T, W)
        s.out = dict(x=x2, h=torch.empty(T, W, dtype=tt, device="cuda"), cache=d["cache"])
        s.keep.append(pr)
        part = lambda heads: C.c_void_p(pr.data_ptr() + 4 * heads * D)  # noqa: E731
        none = (nil, nil, nil, 0, 0, 0, nil, nil, 0, nil, nil, nil)  # no expert slots, no shared expert, no embedding, no added vector
        s.call("ggb_op_residual_layer_norm", dt, d["x"], nil, *none, d["nw"][0], d["nb"][0], 1e-5, W, T, nil, x1, h)
        s.call("ggb_op_linear", dt, d["proj"], N, W, h, W, T, pr, N)
        s.call("ggb_op_head_qkv_store", dt, part(0), part(H), part(H + Gk), N, T, H, Gk, D, D, d["qn"], d["kn"], 1e-5, D, 1, d["cs"], D ** -0.5, pos, d["table"], PAGE,
               d["cache"], qr)
        s.call("ggb_op_masked_attn_gated", dt, qr, d["cache"], d["table"], PAGE, pos, T, H, Gk, D, D, c["window"], 4 if c["window"] else 0, 30.0, nil, part(H + 2 * Gk), N, ao,
               scratch)
        s.call("ggb_op_linear", dt, d["o"], W, HD, ao, HD, T, ya, W)
        s.call("ggb_op_residual_layer_norm", dt, x1, ya, *none, d["nw"][1], d["nb"][1], 1e-5, W, T, nil, x1, h2)
        s.call("ggb_op_linear_act", dt, d["up"], F, W, h2, W, T, 4, act)
        s.call("ggb_op_linear", dt, d["down"], W, F, act, F, T, yf, W)
        s.call("ggb_op_residual_layer_norm", dt, x1, yf, *none, d["nw"][0], d["nb"][0], 1e-5, W, T, nil, x2, s.out["h"])
        torch.cuda.synchronize()
        launch(s)  # kernels are loaded before a capture
        G.sync()
        G.check(L.ggb_capture_begin(), "ggb_capture_begin")
        launch(s)
        s.graph = C.c_void_p()
        G.check(L.ggb_capture_end(C.byref(s.graph)), "ggb_capture_end")
        return s
    if k == "latent":
        d = latent_inputs(c, seed)
        H, R, Dr, Dv = c["heads"], c["rank"], c["rot"], c["vdim"]
        n = c["pos"] + T  # the splits the engine takes
        ns = max(1, min((n + (31 if T <= 8 else 127)) // (32 if T <= 8 else 128), max(1, 296 // T), 64))
        part = torch.empty(int(G.cuda_lib().ggb_latent_attn_scratch_bytes(T, H, R, ns)), dtype=torch.uint8, device="cuda")
        s.out = dict(out=torch.empty(T, H * Dv, dtype=tt, device="cuda"))
        s.call("ggb_op_latent_attn_window", dt, d["qa"], d["cache"], d["table"], PAGE, pos, T, H, R, Dr, c["window"], ns, part)
        s.call("ggb_op_latent_attn_out", dt, part, ns, d["sink"], d["w_uv"], T, H, R, Dv, s.out["out"])
        return s
    d = attention_inputs(c, seed)
    H, Gk, D, Dv = c["heads"], c["kv"], c["dim"], c["vdim"]
    s.out = dict(out=torch.empty(T, H * Dv, dtype=tt, device="cuda"))
    L, maps = G.cuda_lib(), c.get("maps", 1)
    if k == "sigmoid":
        scratch = torch.empty(int(L.ggb_sigmoid_attn_scratch_bytes(H)), dtype=torch.uint8, device="cuda")
        s.call("ggb_op_sigmoid_attn", dt, d["q"], d["cache"], d["table"], PAGE, pos, T, H, Gk, D, Dv, c["window"], d["r1"], d["r2"], d["pb"], s.out["out"], scratch)
        return s
    scratch = torch.empty(int(L.ggb_window_attn_scratch_bytes(H * maps)), dtype=torch.uint8, device="cuda")
    if maps == 1:
        s.call("ggb_op_masked_attn_gated", dt, d["q"], d["cache"], d["table"], PAGE, pos, T, H, Gk, D, Dv, c["window"], c["keep"], c["softcap"], d["sink"], d["gate"], H * Dv,
               s.out["out"], scratch)
    else:
        s.call("ggb_op_diff_attn", dt, d["q"], d["cache"], d["table"], PAGE, pos, T, H, Gk, D, Dv, c["window"], c["keep"], c["softcap"], 0.35, 0.8, 1e-5, d["gate"], H * Dv,
               s.out["out"], scratch)
    return s


def launch(s):
    for name, fn, args in s.calls:
        rc = fn(*args)
        if rc:
            G.check(rc, name)


def run(state):
    s = state
    if s.kind == "decode":
        s.model.decode_step(int(s.tokens[0]), s.pos)
        return {"logits": s.model.logits()}
    if s.kind == "prefill":
        s.model.prefill(s.tokens)
        return {"logits": s.model.prefill_logits(len(s.tokens) - 1)}
    if s.kind == "offload":
        G.check(G.cuda_lib().ggb_mul_mat(*s.args), "ggb_mul_mat")
        return s.dst
    if s.graph is not None:
        G.check(G.cuda_lib().ggb_graph_launch(s.graph), "ggb_graph_launch")
    else:
        launch(s)
    return s.out


# ------------------------------------------------------------------------------------------------------------ what a pass cannot do without
def visible(c):
    """(query, key) pairs of a portion under a causal window with kept first positions"""
    w, keep, n = c["window"], c.get("keep", 0), 0
    for i in range(c["pos"], c["pos"] + c["T"]):
        own = i + 1 if w <= 0 else min(i + 1, w)
        n += own + min(keep, i + 1 - own)
    return n


def work(case):
    c, k = case, case["kind"]
    if k in ("decode", "prefill"):
        E, F, QD, KD = c["embd"], c["ff"], c["heads"] * c["dim"], c["kv"] * c["dim"]
        per = E * (QD + 2 * KD) + QD * E + 3 * E * F
        weights = (c["layers"] * per + c["vocab"] * E) * Q_BYTES[c["q"]]
        if k == "decode":
            kv = 4.0 * KD * c["ctx"] * c["layers"]
            return {"bytes": weights + kv + 4 * c["vocab"], "flops": 2.0 * (c["layers"] * per + c["vocab"] * E) + 4.0 * QD * c["ctx"] * c["layers"]}
        T = c["T"]
        return {"bytes": weights + 4.0 * T * c["vocab"], "flops": 2.0 * T * (c["layers"] * per + c["vocab"] * E) + 2.0 * QD * T * (T + 1) * c["layers"]}
    if k in ("offload", "kquant"):
        a = 34 / 32 if k == "offload" else 4
        return {"bytes": c["rows"] * c["cols"] * Q_BYTES[c["q"]] + c["T"] * c["cols"] * a + 4.0 * c["T"] * c["rows"], "flops": 2.0 * c["rows"] * c["cols"] * c["T"]}
    if k == "delta":
        T, H, D, Dv, Gk = c["T"], c["heads"], c["dim"], c["vdim"], c["heads"] if c["rule"] == "lightning" else c["kv"]
        a = {"head": 2 * H, "channel": H + H * D, "lightning": 0}[c["rule"]]
        return {"bytes": 4.0 * (T * (2 * Gk * D + H * Dv + a + H * Dv) + 2 * H * D * Dv), "flops": T * H * D * Dv * (5.0 if c["rule"] == "lightning" else 8.0)}
    es, T = KIND_OF[c["dt"]][2], c["T"]
    if k == "linear":
        return {"bytes": float(es * (c["N"] * c["K"] + T * c["K"]) + 4 * T * c["N"]), "flops": 2.0 * T * c["N"] * c["K"]}
    if k == "experts":
        W, F, E = c["width"], c["ff"], c["experts"]
        used = min(E, T * c["top"])
        return {"bytes": float(used * 2 * W * F * es + T * W * (es + 4) + 4 * E * W), "flops": 4.0 * T * c["top"] * W * F + 2.0 * T * W * E}
    if k == "layer":
        W, H, Gk, D, F = c["width"], c["heads"], c["kv"], c["dim"], c["ff"]
        mats = (2 * H + 2 * Gk) * D * W + H * D * W + 2 * F * W
        v = visible(dict(c, keep=4 if c["window"] else 0))
        return {"bytes": float(es * (mats + 2 * Gk * D * (v / T + T)) + 4 * T * W * 2), "flops": 2.0 * T * mats + 4.0 * H * D * v}
    seen = c["pos"] + T if c["window"] <= 0 else min(c["pos"] + T, c["window"] + T + c.get("keep", 0))
    if k == "latent":
        R, Dr, H, Dv = c["rank"], c["rot"], c["heads"], c["vdim"]
        return {"bytes": float(es * (seen * (R + Dr) + H * Dv * R + T * H * Dv) + 4 * T * H * (R + Dr)),
                "flops": 2.0 * H * visible(c) * (2 * R + Dr) + 2.0 * T * H * R * Dv}
    maps, H, Gk, D, Dv = c.get("maps", 1), c["heads"], c["kv"], c["dim"], c["vdim"]
    return {"bytes": float(es * (seen * Gk * (maps * D + Dv) + T * H * Dv) + 4 * T * H * (maps * D + (Dv if c.get("gate") else 0))),
            "flops": 2.0 * H * maps * visible(c) * (D + Dv)}


def tolerance(case):
    """Integer dots with one stated order are bit-identical; sums of fp32 products 2e-5; results that leave in bf16, or go through a bf16
    intermediate, a few of its roundings."""
    k = case["kind"]
    if k in ("offload", "kquant", "decode"):
        return "exact"
    if k == "prefill":
        return {"rel": 0.03, "max": 0.3}
    if k == "delta":
        return {"rel": 2e-5, "max": 2e-3}
    if k == "linear" or case["dt"] == "f32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 4e-3, "max": 0.1}


# ------------------------------------------------------------------------------------------------------------ the results in 64 bits
def softmax_heads(q, K, V, vis, softcap, sink):
    s = q @ K.T
    if softcap > 0:
        s = softcap * torch.tanh(s / softcap)
    s = s.masked_fill(~vis, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.expand(s.shape[0], 1)], 1)
    p = torch.softmax(s, 1)
    return p[:, :V.shape[0]] @ V


def mask_of(pos, T, window, keep):
    i = torch.arange(pos, pos + T, device="cuda")[:, None]
    j = torch.arange(pos + T, device="cuda")[None, :]
    vis = j <= i
    if window > 0:
        vis = vis & ((i - j < window) | (j < keep))
    return i, j, vis


def exact_attention(c, seed):
    d = attention_inputs(c, seed)
    maps, H, Gk, D, Dv, T = c.get("maps", 1), c["heads"], c["kv"], c["dim"], c["vdim"], c["T"]
    n = c["pos"] + T
    rows = rows_of(d["cache"], d["table"], n).double()
    K = rows[:, :Gk * maps * D].reshape(n, Gk, maps, D)
    V = rows[:, Gk * maps * D:Gk * (maps * D + Dv)].reshape(n, Gk, Dv)
    i, j, vis = mask_of(c["pos"], T, c["window"], c.get("keep", 0))
    q, out = d["q"].double(), torch.empty(T, H, Dv, dtype=torch.float64, device="cuda")
    for h in range(H):
        g = h // (H // Gk)
        if c["kind"] == "sigmoid":
            z = q[:, h, 0] @ K[:, g, 0].T - d["r1"][h].double() * torch.log1p(d["r2"][h].double() * (i - j).clamp(min=0)) + d["pb"][h].double()
            out[:, h] = (torch.sigmoid(z) * vis) @ V[:, g]
            continue
        o = [softmax_heads(q[:, h, m], K[:, g, m], V[:, g], vis, c["softcap"], d["sink"][h].double().reshape(1, 1) if d["sink"] is not None else None) for m in range(maps)]
        if maps == 2:
            o[0] = o[0] - float(np.float32(0.35)) * o[1]
            o[0] = o[0] / torch.sqrt((o[0] ** 2).mean(1, keepdim=True) + 1e-5) * 0.8
        out[:, h] = o[0]
    out = out.reshape(T, H * Dv)
    if d["gate"] is not None:
        out = out * torch.sigmoid(d["gate"].double())
    return {"out": out}


def exact_latent(c, seed):
    d = latent_inputs(c, seed)
    H, R, Dr, Dv, T = c["heads"], c["rank"], c["rot"], c["vdim"], c["T"]
    rows = rows_of(d["cache"], d["table"], c["pos"] + T).double()[:, :R + Dr]
    _, _, vis = mask_of(c["pos"], T, c["window"], 0)
    out = torch.empty(T, H, Dv, dtype=torch.float64, device="cuda")
    for h in range(H):
        o = softmax_heads(d["qa"][:, h].double(), rows, rows[:, :R], vis, 0.0, d["sink"][h].double().reshape(1, 1))
        out[:, h] = o @ d["w_uv"].double()[h * Dv:(h + 1) * Dv].T
    return {"out": out.reshape(T, H * Dv)}


def exact_experts(c, seed):
    d = experts_inputs(c, seed)
    h = d["h"].double()
    w, idx = (h @ d["router"].double().T + d["bias"].double()).topk(c["top"], 1)
    w = torch.softmax(w, 1)
    y = torch.zeros(c["T"], c["width"], dtype=torch.float64, device="cuda")
    for e in range(c["experts"]):
        t, s = (idx == e).nonzero(as_tuple=True)
        if t.numel():
            y.index_add_(0, t, w[t, s, None] * (torch.nn.functional.gelu(h[t] @ d["up"][e].double().T) @ d["down"][e].double().T))
    return {"y": y}


def exact_layer(c, seed):
    d = {k: v.double() if v.is_floating_point() else v for k, v in layer_inputs(c, seed).items()}
    T, W, H, Gk, D = c["T"], c["width"], c["heads"], c["kv"], c["dim"]
    n = c["pos"] + T

    def norm(x, k):
        x = x - x.mean(1, keepdim=True)
        return x / torch.sqrt((x ** 2).mean(1, keepdim=True) + 1e-5) * d["nw"][k] + d["nb"][k]

    def head(x, w):  # norm per head, then the halves turn
        x = x / torch.sqrt((x ** 2).mean(-1, keepdim=True) + 1e-5) * w
        cs = d["cs"][c["pos"]:n, None]
        u, v = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([u * cs[..., 0] - v * cs[..., 1], v * cs[..., 0] + u * cs[..., 1]], -1)

    pr = (norm(d["x"], 0) @ d["proj"].T).reshape(T, 2 * H + 2 * Gk, D)
    q, kk, v, gate = head(pr[:, :H], d["qn"]) * D ** -0.5, head(pr[:, H:H + Gk], d["kn"]), pr[:, H + Gk:H + 2 * Gk], pr[:, H + 2 * Gk:]
    j = torch.arange(c["pos"], n, device="cuda")
    d["cache"][d["table"].long()[j // PAGE] * PAGE + j % PAGE, :2 * Gk * D] = torch.cat([kk, v], 1).reshape(T, -1)
    rows = rows_of(d["cache"], d["table"], n)
    _, _, vis = mask_of(c["pos"], T, c["window"], 4 if c["window"] else 0)
    ao = torch.stack([softmax_heads(q[:, h], rows[:, (h // (H // Gk)) * D:][:, :D], rows[:, (Gk + h // (H // Gk)) * D:][:, :D], vis, 30.0, None) for h in range(H)], 1)
    x = d["x"] + (ao * torch.sigmoid(gate)).reshape(T, H * D) @ d["o"].T
    x = x + torch.nn.functional.gelu(norm(x, 1) @ d["up"].T) @ d["down"].T
    return {"x": x, "h": norm(x, 0), "cache": d["cache"]}


def exact_delta(c, seed):
    d = delta_inputs(c, seed)
    T, H, Gk, D, Dv = c["T"], c["heads"], d["Gk"], c["dim"], c["vdim"]
    x, S = d["x"].double(), d["state"].double()
    q, kk = (x[:, o:o + Gk * D].reshape(T, Gk, D).repeat_interleave(H // Gk, 1) for o in (0, Gk * D))
    v = x[:, 2 * Gk * D:].reshape(T, H, Dv)
    if c["rule"] == "lightning":
        silu = torch.nn.functional.silu
        q, kk, v = silu(q), silu(kk), silu(v)
        g, beta = d["decay"].double().expand(T, H)[..., None], None
    else:
        q = q / torch.sqrt((q ** 2).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
        kk = kk / torch.sqrt((kk ** 2).sum(-1, keepdim=True) + 1e-6)
        beta = torch.sigmoid(d["b"].double())
        a = torch.nn.functional.softplus(d["a"].double() + d["dt_bias"].double()).reshape(T, H, -1)
        g = torch.exp(-torch.exp(d["A_log"].double())[:, None] * a)
    o = torch.empty(T, H, Dv, dtype=torch.float64, device="cuda")
    for t in range(T):
        S = S * g[t][..., None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, kk[t]))
        S = S + kk[t][..., None] * u[:, None]
        o[t] = torch.einsum("hdv,hd->hv", S, q[t])
    return {"o": o.reshape(T, H * Dv), "state": S}


def blocks_q(q, b):
    """weights of Q4_0 / Q8_0 blocks [..., 18 | 34] in 64 bits"""
    d = b[..., 0:2].contiguous().view(torch.float16).double()
    if q == "q8_0":
        return b[..., 2:].contiguous().view(torch.int8).double() * d
    return torch.cat([(b[..., 2:] & 15).double() - 8, (b[..., 2:] >> 4).double() - 8], -1) * d


def exact_offload(c, seed):
    w, a = (torch.from_numpy(x).cuda() for x in offload_inputs(c, seed))
    nb = c["cols"] // 32
    return blocks_q("q8_0", a.reshape(c["T"], nb, 34)).reshape(c["T"], -1) @ blocks_q(c["q"], w.reshape(c["rows"], nb, -1)).reshape(c["rows"], -1).T


def exact_kquant(c, seed):
    raw, x = kquant_inputs(c, seed)
    nb = c["cols"] // 256
    x = x.reshape(c["T"], nb, 256)
    top = x.gather(2, x.abs().argmax(2, keepdim=True))
    isc = -128.0 / top  # the row as the format has it: int8 codes and one scale a block
    x = torch.round(isc * x).clamp(max=127).double() * (1.0 / isc).double()
    y = torch.empty(c["T"], c["rows"], dtype=torch.float64, device="cuda")
    for r in range(0, c["rows"], 16384):
        b = raw[r:r + 16384].reshape(-1, nb, raw.shape[1] // nb)
        if c["q"] == "q4_k":
            d, dmin = (b[..., o:o + 2].contiguous().view(torch.float16).double() for o in (0, 2))
            p, qs = b[..., 4:16].int(), b[..., 16:].reshape(*b.shape[:2], 4, 32)
            sc = torch.cat([p[..., 0:4] & 63, (p[..., 8:12] & 15) | ((p[..., 0:4] >> 6) << 4)], -1).double()
            mn = torch.cat([p[..., 4:8] & 63, (p[..., 8:12] >> 4) | ((p[..., 4:8] >> 6) << 4)], -1).double()
            codes = torch.stack([qs & 15, qs >> 4], -2).reshape(*b.shape[:2], 8, 32).double()
            w = d[..., None] * sc[..., None] * codes - dmin[..., None] * mn[..., None]
        else:
            ql, qh = b[..., :128].reshape(*b.shape[:2], 2, 64).int(), b[..., 128:192].reshape(*b.shape[:2], 2, 32).int()
            sc, d = b[..., 192:208].contiguous().view(torch.int8).double(), b[..., 208:210].contiguous().view(torch.float16).double()
            codes = torch.stack([(ql[..., :32] & 15) | ((qh & 3) << 4), (ql[..., 32:] & 15) | (((qh >> 2) & 3) << 4), (ql[..., :32] >> 4) | (((qh >> 4) & 3) << 4),
                                 (ql[..., 32:] >> 4) | (((qh >> 6) & 3) << 4)], -2).reshape(*b.shape[:2], 16, 16)
            w = d[..., None] * sc[..., None] * (codes - 32).double()
        y[:, r:r + 16384] = x.reshape(c["T"], -1) @ w.reshape(b.shape[0], -1).T
    return {"y": y}


def synth(seed, tensor, first, n, sigma):
    """the library's counter-based synthetic numbers: splitmix64 of a key and the index, four 16-bit fields added up"""
    mask = (1 << 64) - 1

    def mix(x):
        x = (x + 0x9E3779B97F4A7C15) & mask
        x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & mask
        x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & mask
        return x ^ (x >> 31)

    def wrap(v):
        return v - (1 << 64) if v >> 63 else v

    key = mix((seed + tensor * 0xD1B54A32D192ED03) & mask)
    x = torch.arange(first, first + n, dtype=torch.int64, device="cuda") + wrap((key + 0x9E3779B97F4A7C15) & mask)
    x = (x ^ ((x >> 30) & ((1 << 34) - 1))) * wrap(0xBF58476D1CE4E5B9)
    x = (x ^ ((x >> 27) & ((1 << 37) - 1))) * wrap(0x94D049BB133111EB)
    x = x ^ ((x >> 31) & ((1 << 33) - 1))
    total = (x & 0xFFFF) + ((x >> 16) & 0xFFFF) + ((x >> 32) & 0xFFFF) + ((x >> 48) & 0xFFFF) - 131070
    unit = float(np.float32(sigma) * np.float32(np.float32(1.0) / np.float32(37837.2274)))
    return total.float() * unit


def synth_matrix(c, seed, tensor, rows, cols, row0=0):
    """rows of a synthetic matrix as the quantised format holds them, in 64 bits"""
    v = synth(seed, tensor, row0 * cols, rows * cols, 0.02).reshape(-1, 32)
    if c["q"] == "q4_0":
        d = v.gather(1, v.abs().argmax(1, keepdim=True)) / -8.0
        codes = torch.floor(v * (1.0 / d) + 8.5).clamp(max=15) - 8
    else:
        d = v.abs().amax(1, keepdim=True) / 127.0
        z = v * (1.0 / d)
        codes = torch.sign(z) * torch.floor(z.abs() + 0.5)
    return (codes.double() * d.half().double()).reshape(rows, cols)


def exact_gemma(c, seed):
    """the forward pass in 64 bits on the quantised weights (activations are not rounded at all)"""
    cfg = gemma_config(c, seed)
    ws, E, F, H, Gk, D, decode = cfg.seed, c["embd"], c["ff"], c["heads"], c["kv"], c["dim"], c["kind"] == "decode"
    tokens = torch.from_numpy(prompt_of(c, seed)).long().cuda()
    T, pos = len(tokens), c["ctx"] - 1 if decode else 0

    def norm(x, tensor):
        return x / torch.sqrt((x ** 2).mean(1, keepdim=True) + 1e-6) * (1.0 + synth(ws, tensor, 0, E, 0.02).double())

    p = torch.arange(pos, pos + T, device="cuda", dtype=torch.float64)[:, None, None]
    ang = p * 10000.0 ** (-torch.arange(D // 2, device="cuda", dtype=torch.float64) * 2 / D)

    def rope(x):
        u, v = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([u * ang.cos() - v * ang.sin(), u * ang.sin() + v * ang.cos()], -1)

    x = torch.cat([synth_matrix(c, ws, 0, 1, E, int(t)) for t in tokens]) * math.sqrt(E)
    _, _, vis = mask_of(pos, T, 0, 0)
    for layer in range(c["layers"]):
        mat = lambda i, rows, cols: synth_matrix(c, ws, 2 + 9 * layer + i, rows, cols)  # noqa: B023, E731
        h = norm(x, 2 + 9 * layer)
        q, k, v = ((h @ mat(1 + i, n * D, E).T).reshape(T, n, D) for i, n in enumerate((H, Gk, Gk)))
        q, k = rope(q) * D ** -0.5, rope(k)
        if decode:
            old = [synth(seed, 2 * layer + i, 0, c["ctx"] * Gk * D, 1.0).half().double().reshape(c["ctx"], Gk, D)[:pos] for i in range(2)]
            k, v = torch.cat([old[0], k]), torch.cat([old[1], v])
        ao = torch.stack([softmax_heads(q[:, i], k[:, i // (H // Gk)], v[:, i // (H // Gk)], vis, 0.0, None) for i in range(H)], 1)
        x = x + ao.reshape(T, H * D) @ mat(4, E, H * D).T
        h = norm(x, 2 + 9 * layer + 5)
        x = x + (torch.nn.functional.gelu(h @ mat(6, F, E).T, approximate="tanh") * (h @ mat(7, F, E).T)) @ mat(8, E, F).T
    h = norm(x, 1)[-1:]
    return {"logits": torch.cat([h @ synth_matrix(c, ws, 0, min(32768, c["vocab"] - r), E, r).T for r in range(0, c["vocab"], 32768)], 1).reshape(-1)}


def exact(case, seed):
    c = case
    if c["kind"] == "linear":
        d = linear_inputs(c, seed)
        return {"c": d["a"].double() @ d["w"].double().T}
    return {"offload": exact_offload, "kquant": exact_kquant, "decode": exact_gemma, "prefill": exact_gemma, "experts": exact_experts, "layer": exact_layer,
            "attention": exact_attention, "sigmoid": exact_attention, "latent": exact_latent, "delta": exact_delta}[c["kind"]](c, seed)
