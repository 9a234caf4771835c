"""The tensor-core form of attention over portions (csrc/tile_attention.cuh) against float64, at the edges of its tiles: 128 query rows
(tokens x heads of a key head, or half as many with two maps) and 64 keys.  Both sides see the same bf16 cache and fp32 queries; the
result differs by its rounding to bf16, at most 2^-9 of a value, plus fp32 sums (1e-6): a relative error (2-norm) of 2.5e-3 at most."""
import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, f32, from_dt, i32, ptr, release, zeros

pytestmark = pytest.mark.gpu
LIMIT = 2.5e-3


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def inputs(gpu, dt, H, G, D, Dv, maps, pos, T, page, seed, scale):
    r = np.random.default_rng(seed)
    n, ld = pos + T, int(gpu.cuda_lib().ggb_window_cache_ld(G, D * maps, Dv))
    pages = (n + page - 1) // page
    table = r.permutation(pages + 2)[:pages].astype(np.int32)
    cache, raw = as_dt(BF16, r.standard_normal(((pages + 2) * page, ld)))
    rows = cache[table[np.arange(n) // page].astype(np.int64) * page + np.arange(n) % page]
    q = f32(r.standard_normal((T, H, maps, D)) * scale)
    if dt == F32:
        raw = f32(cache)
    K = rows[:, :G * maps * D].reshape(n, G, maps, D)
    V = rows[:, G * maps * D:G * (maps * D + Dv)].reshape(n, G, Dv)
    return r, q, K, V, dev(gpu, raw), dev(gpu, table), dev(gpu, i32([pos]))


def seen(pos, T, window, keep, chunked):
    i, j = np.arange(pos, pos + T)[:, None], np.arange(pos + T)[None]
    if window <= 0:
        return j <= i
    lo = i - i % window if chunked else i - window + 1
    return (j <= i) & ((j >= lo) | (j < keep))


def soft(q, K, V, vis, cap, sink):
    s = q @ K.T
    s = np.where(vis, cap * np.tanh(s / cap) if cap else s, -np.inf)
    m = np.maximum(s.max(1), sink if sink is not None else -np.inf)
    e = np.exp(s - m[:, None])
    return (e @ V) / (e.sum(1) + (np.exp(sink - m) if sink is not None else 0.0))[:, None]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# H, Gk, D, Dv, T, pos, page, window, keep, chunked, cap, scale, sink, gate
SOFT = [(1, 1, 16, 16, 32, 0, 64, 0, 0, 0, 0.0, 0.3, 1, 0), (4, 1, 64, 64, 33, 31, 64, 0, 0, 0, 0.0, 0.1, 0, 1), (3, 1, 80, 112, 129, 64, 7, 65, 1, 0, 30.0, 0.2, 1, 1),
        (2, 2, 128, 128, 128, 0, 64, 64, 0, 0, 30.0, 1.0, 0, 0), (16, 1, 128, 128, 40, 500, 64, 300, 70, 0, 2.0, 0.5, 0, 1), (6, 2, 192, 128, 127, 129, 16, 100, 0, 1, 0.0, 0.1, 0, 0),
        (5, 5, 48, 96, 200, 3, 64, 1, 130, 0, 0.0, 0.3, 1, 0), (8, 8, 96, 80, 300, 700, 64, 128, 64, 0, 0.0, 2.0, 0, 1), (128, 1, 32, 32, 35, 66, 64, 0, 0, 0, 5.0, 0.4, 0, 0),
        # keys of three blocks of 64 with values of one, the most that shared memory holds (192 with 128 above runs on the CUDA cores)
        (6, 2, 192, 64, 127, 129, 16, 100, 0, 1, 0.0, 0.1, 0, 0), (4, 1, 176, 48, 70, 30, 64, 0, 0, 0, 30.0, 0.5, 1, 1)]


# clusters of two, four and eight CTAs that share key tiles: CTAs of few tiles, of a part or none for some of them, rows that see nothing of a part, a window of a part
SOFT += [(4, 1, 64, 64, 385, 0, 64, 0, 0, 0, 30.0, 0.5, 1, 1), (2, 1, 128, 128, 800, 90, 64, 0, 0, 0, 0.0, 1.0, 0, 0), (3, 1, 32, 48, 900, 5, 16, 400, 70, 0, 0.0, 0.3, 0, 1),
         (6, 3, 16, 80, 1000, 130, 64, 768, 0, 0, 2.0, 0.4, 1, 0), (1, 1, 64, 128, 777, 500, 64, 390, 0, 1, 0.0, 0.3, 0, 0),
         (4, 1, 64, 64, 640, 0, 64, 0, 0, 0, 30.0, 0.5, 1, 1), (2, 2, 48, 32, 639, 200, 64, 0, 0, 0, 0.0, 0.5, 0, 0), (1, 1, 64, 128, 777, 500, 64, 650, 0, 1, 0.0, 0.3, 0, 0),
         (1, 1, 64, 64, 1536, 0, 64, 0, 0, 0, 30.0, 0.5, 1, 1), (1, 1, 32, 48, 1750, 333, 16, 0, 0, 0, 0.0, 1.0, 0, 0), (1, 1, 16, 80, 1700, 900, 64, 1600, 70, 0, 0.0, 0.3, 0, 1)]


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("H,Gk,D,Dv,T,pos,page,window,keep,chunked,cap,scale,sink,gate", SOFT)
def test_soft_max_heads(gpu, dt, H, Gk, D, Dv, T, pos, page, window, keep, chunked, cap, scale, sink, gate):
    G = Gk
    r, q, K, V, cache, table, pos0 = inputs(gpu, dt, H, G, D, Dv, 1, pos, T, page, D + T, scale)
    s, g = r.standard_normal(H), r.standard_normal((T, H * Dv))
    out = zeros(gpu, T * H * Dv * (2 if dt == BF16 else 4))
    lib = gpu.cuda_lib()
    if chunked:
        gpu.check(lib.ggb_op_masked_attn(dt, dev(gpu, q).ptr, cache.ptr, table.ptr, page, pos0.ptr, T, H, G, D, Dv, window, 1, cap, None, out.ptr, None), "attn")
    else:
        gpu.check(lib.ggb_op_masked_attn_gated(dt, dev(gpu, q).ptr, cache.ptr, table.ptr, page, pos0.ptr, T, H, G, D, Dv, window, keep, cap, ptr(dev(gpu, f32(s)) if sink else None),
                                               ptr(dev(gpu, f32(g)) if gate else None), H * Dv, out.ptr, None), "attn")
    vis = seen(pos, T, window, keep, chunked)
    want = np.stack([soft(q[:, h, 0].astype(np.float64), K[:, h // (H // G), 0], V[:, h // (H // G)], vis, cap, f32(s)[h].astype(np.float64) if sink else None) for h in range(H)], 1)
    want = want.reshape(T, H * Dv) / (1.0 + np.exp(-f32(g).astype(np.float64)) if gate else 1.0)
    assert rel(from_dt(dt, out, (T, H * Dv)), want) < (LIMIT if dt == BF16 else 1e-5)


@pytest.mark.parametrize("H,Gk,D,Dv,T,pos,window,keep,cap", [(2, 1, 16, 16, 32, 0, 0, 0, 0.0), (4, 2, 64, 128, 65, 63, 64, 3, 30.0), (3, 3, 128, 128, 64, 200, 0, 0, 2.0), (64, 1, 32, 48, 33, 90, 70, 65, 0.0),
                                                                   (2, 1, 64, 64, 800, 300, 0, 0, 30.0), (1, 1, 32, 128, 450, 0, 400, 9, 0.0), (2, 1, 64, 64, 640, 0, 0, 0, 0.0), (1, 1, 32, 128, 1600, 70, 700, 9, 0.0)])
def test_differential_heads(gpu, H, Gk, D, Dv, T, pos, window, keep, cap):
    G = Gk
    r, q, K, V, cache, table, pos0 = inputs(gpu, BF16, H, G, D, Dv, 2, pos, T, 64, D + T, 0.3)
    out, lam, eps = zeros(gpu, T * H * Dv * 2), 0.4, 1e-5
    gpu.check(gpu.cuda_lib().ggb_op_diff_attn(BF16, dev(gpu, q).ptr, cache.ptr, table.ptr, 64, pos0.ptr, T, H, G, D, Dv, window, keep, cap, lam, 0.7, eps, None, 0, out.ptr, None), "attn")
    vis, q = seen(pos, T, window, keep, 0), q.astype(np.float64)
    o = np.stack([soft(q[:, h, 0], K[:, h // (H // G), 0], V[:, h // (H // G)], vis, cap, None) - np.float32(lam) * soft(q[:, h, 1], K[:, h // (H // G), 1], V[:, h // (H // G)], vis, cap, None)
                  for h in range(H)], 1)
    o = o / np.sqrt((o ** 2).mean(-1, keepdims=True) + eps) * 0.7
    assert rel(from_dt(BF16, out, (T, H, Dv)), o) < LIMIT


@pytest.mark.parametrize("H,Gk,D,Dv,T,pos,window,page,bare", [(1, 1, 16, 16, 32, 0, 0, 64, 0), (4, 1, 64, 64, 33, 31, 0, 5, 0), (16, 1, 128, 128, 129, 64, 65, 64, 0), (6, 2, 80, 96, 200, 700, 128, 64, 0), (4, 1, 64, 80, 800, 200, 0, 64, 0), (2, 2, 32, 32, 390, 0, 0, 16, 1), (1, 1, 64, 64, 1600, 0, 0, 64, 0), (1, 1, 48, 80, 1750, 500, 0, 16, 0),
                                                            (64, 1, 48, 32, 40, 100, 0, 64, 0), (3, 3, 128, 128, 128, 0, 1, 64, 1)])
def test_sigmoid_heads(gpu, H, Gk, D, Dv, T, pos, window, page, bare):
    G = Gk
    r, q, K, V, cache, table, pos0 = inputs(gpu, BF16, H, G, D, Dv, 1, pos, T, page, D + T, 1.5)
    r1, r2, pb = f32(r.uniform(0.2, 1.0, H)), f32(r.uniform(0.1, 1.5, H)), f32(r.uniform(-2.5, 0.0, H))
    d = [None if bare else dev(gpu, a) for a in (r1, r2, pb)]
    out = zeros(gpu, T * H * Dv * 2)
    gpu.check(gpu.cuda_lib().ggb_op_sigmoid_attn(BF16, dev(gpu, q).ptr, cache.ptr, table.ptr, page, pos0.ptr, T, H, G, D, Dv, window, *(ptr(x) for x in d), out.ptr, None), "attn")
    vis, dist = seen(pos, T, window, 0, 0), np.maximum(np.arange(pos, pos + T)[:, None] - np.arange(pos + T)[None], 0)
    want = []
    for h in range(H):
        z = q[:, h, 0].astype(np.float64) @ K[:, h // (H // G), 0].T
        if not bare:
            z = z - np.float64(r1[h]) * np.log1p(np.float64(r2[h]) * dist) + np.float64(pb[h])
        want.append((vis / (1.0 + np.exp(-z))) @ V[:, h // (H // G)])
    assert rel(from_dt(BF16, out, (T, H, Dv)), np.stack(want, 1)) < LIMIT


def attend(gpu, kind, q, cache, table, pos0, T, pos, H, G, D, Dv, cap=0.0, window=0, keep=0, sink=None, gate=None, offsets=None):
    """one call of soft-max, differential or sigmoid heads over a bf16 cache: [T][H][Dv]"""
    lib, out = gpu.cuda_lib(), zeros(gpu, T * H * Dv * 2)
    head = (BF16, dev(gpu, q).ptr, cache.ptr, table.ptr, 64, pos0.ptr, T, H, G, D, Dv, window)
    g, s = ptr(dev(gpu, f32(gate)) if gate is not None else None), ptr(dev(gpu, f32(sink)) if sink is not None else None)
    if kind == "soft":
        gpu.check(lib.ggb_op_masked_attn_gated(*head, keep, cap, s, g, H * Dv, out.ptr, None), "attn")
    elif kind == "diff":
        gpu.check(lib.ggb_op_diff_attn(*head, keep, cap, 0.4, 0.7, 1e-5, g, H * Dv, out.ptr, None), "attn")
    else:
        gpu.check(lib.ggb_op_sigmoid_attn(*head, *(ptr(dev(gpu, f32(o))) for o in (np.zeros((3, H)) if offsets is None else offsets)), out.ptr, None), "attn")
    return from_dt(BF16, out, (T, H, Dv))


@pytest.mark.parametrize("kind,cap", [("soft", 0.0), ("soft", 30.0), ("diff", 0.0), ("sigmoid", 0.0)])
@pytest.mark.parametrize("where", ["query", "key", "value", "gate"])
def test_nan_stays_nan_and_where_it_is(gpu, kind, cap, where):
    if kind == "sigmoid" and where == "gate":
        pytest.skip("these heads have no gate")
    H, G, D, Dv, T, pos, maps = 4, 2, 64, 64, 70, 90, 2 if kind == "diff" else 1
    r, q, K, V, cache, table, pos0 = inputs(gpu, BF16, H, G, D, Dv, maps, pos, T, 64, 3, 0.3)
    gate = r.standard_normal((T, H * Dv)) if kind != "sigmoid" else None
    call = lambda: attend(gpu, kind, q, cache, table, pos0, T, pos, H, G, D, Dv, cap, gate=gate)  # noqa: E731
    want = call()
    assert np.isfinite(want).all()
    bad = np.zeros((T, H, Dv), bool)
    t0, g, c = 33, 1, 5  # a token, a key head, a coordinate
    if where == "query":
        q[t0, 2, maps - 1, c] = np.nan
        bad[t0, 2] = True
    elif where == "gate":
        gate[t0, 2 * Dv + c] = np.nan
        bad[t0, 2, c] = True
    else:
        raw, tab = cache.download(np.uint16).reshape(-1, int(gpu.cuda_lib().ggb_window_cache_ld(G, D * maps, Dv))), table.download(np.int32)
        raw[tab[(pos + t0) // 64] * 64 + (pos + t0) % 64, (g * maps * D if where == "key" else G * maps * D + g * Dv) + c] = 0x7fc0
        cache.upload(raw)
        bad[t0:, 2 * g:2 * g + 2] = True
        if where == "value" and kind != "diff":  # one coordinate; the norm of a differential head reaches all of them
            bad[:, :, np.arange(Dv) != c] = False
    got = call()
    assert np.isnan(got[bad]).all()
    if where == "value":  # tokens that do not see it, and the other coordinates: finite numbers by another order of sums
        assert rel(got[~bad], want[~bad]) < LIMIT
    else:
        assert (got[~bad] == want[~bad]).all()


def plain_heads(kind, q, K, V, vis, cap, offsets, dist):
    """soft-max, differential or sigmoid heads in float64, only visible keys taking part (0 times an invisible infinity is nothing)"""
    T, H, maps, _ = q.shape
    out = np.empty((T, H, V.shape[2]))
    for t in range(T):
        j = vis[t]
        for h in range(H):
            g, o = h // (H // K.shape[1]), []
            for mp in range(maps):
                s = K[j, g, mp].astype(np.float64) @ q[t, h, mp].astype(np.float64)
                if kind == "sigmoid":
                    p = 1.0 / (1.0 + np.exp(-(s - offsets[0][h] * np.log1p(offsets[1][h] * dist[t, j]) + offsets[2][h])))
                else:
                    s = cap * np.tanh(s / cap) if cap else s
                    p = np.exp(s - s.max())
                    p = p / p.sum()
                o.append(p @ V[j, g])
            if maps == 2:
                o = [o[0] - np.float32(0.4) * o[1]]
                o[0] = o[0] / np.sqrt((o[0] ** 2).mean() + 1e-5) * 0.7
            out[t, h] = o[0]
    return out


@pytest.mark.parametrize("kind,cap,window,keep", [("soft", 0.0, 0, 0), ("soft", 30.0, 50, 3), ("diff", 0.0, 0, 0), ("diff", 30.0, 0, 0), ("sigmoid", 0.0, 0, 0), ("sigmoid", 0.0, 40, 0)])
@pytest.mark.parametrize("where", ["query", "key", "value"])
def test_infinities_as_plain_arithmetic_has_them(gpu, kind, cap, window, keep, where):
    H, G, D, Dv, T, pos, maps = 6, 2, 48, 80, 45, 30, 2 if kind == "diff" else 1
    r, q, K, V, cache, table, pos0 = inputs(gpu, BF16, H, G, D, Dv, maps, pos, T, 64, 7, 0.3)
    K, V = K.copy(), V.copy()
    offsets = np.float32([r.uniform(0.2, 1.0, H), r.uniform(0.1, 1.5, H), r.uniform(-2.5, 0.0, H)])
    ld = int(gpu.cuda_lib().ggb_window_cache_ld(G, D * maps, Dv))
    raw, tab = cache.download(np.uint16).reshape(-1, ld), table.download(np.int32)
    q[5, 1, 0, 3] = np.float32(1.5)  # a query number whose second and third parts are zero
    for at, c, v in [(1, 3, np.inf), (pos + 7, 9, -np.inf), (pos + 33, 3, np.inf)]:  # first page, inside the portion
        slot = tab[at // 64] * 64 + at % 64
        if where == "key":
            K[at, 1, 0, c] = v
            raw[slot, maps * D + c] = 0x7f80 if v > 0 else 0xff80
        elif where == "value":
            V[at, 0, c] = v
            raw[slot, G * maps * D + c] = 0x7f80 if v > 0 else 0xff80
        elif at >= pos:
            q[at - pos, 4, 0, c] = v
    cache.upload(raw)
    vis = seen(pos, T, window, keep, 0)
    dist = np.maximum(np.arange(pos, pos + T)[:, None] - np.arange(pos + T)[None], 0)
    got = attend(gpu, kind, q, cache, table, pos0, T, pos, H, G, D, Dv, cap, window, keep, offsets=offsets)
    with np.errstate(invalid="ignore", over="ignore"):
        want = plain_heads(kind, q, K, V, vis, cap, offsets.astype(np.float64), dist)
    assert np.isfinite(want).any() and (np.isnan(got) == np.isnan(want)).all() and (got[np.isinf(want)] == want[np.isinf(want)]).all()
    ok = np.isfinite(want)
    assert np.isfinite(got[ok]).all() and rel(got[ok], want[ok]) < LIMIT


@pytest.mark.parametrize("kind,cap,window,keep,H,Gk,T", [("soft", 30.0, 0, 0, 6, 2, 450), ("soft", 0.0, 390, 9, 6, 2, 450), ("diff", 0.0, 0, 0, 6, 2, 450), ("sigmoid", 0.0, 0, 0, 6, 2, 450),
                                                        ("soft", 30.0, 0, 0, 6, 2, 700), ("soft", 0.0, 650, 9, 6, 2, 900), ("diff", 0.0, 0, 0, 6, 2, 700), ("soft", 0.0, 0, 0, 1, 1, 1600),
                                                        ("sigmoid", 0.0, 0, 0, 1, 1, 1600)])
@pytest.mark.parametrize("where", ["query", "key", "value"])
def test_infinities_in_the_tiles_of_a_cluster(gpu, kind, cap, window, keep, H, Gk, T, where):
    """the same where several CTAs have the key tiles: a row that is not finite in one of them is computed once more over all of its keys"""
    G, D, Dv, pos, maps = Gk, 48, 80, 260, 2 if kind == "diff" else 1
    r, q, K, V, cache, table, pos0 = inputs(gpu, BF16, H, G, D, Dv, maps, pos, T, 64, 7, 0.3)
    K, V = K.copy(), V.copy()
    offsets = np.float32([r.uniform(0.2, 1.0, H), r.uniform(0.1, 1.5, H), r.uniform(-2.5, 0.0, H)])
    ld = int(gpu.cuda_lib().ggb_window_cache_ld(G, D * maps, Dv))
    raw, tab = cache.download(np.uint16).reshape(-1, ld), table.download(np.int32)
    q[5, min(1, H - 1), 0, 3] = np.float32(1.5)  # a query number whose second and third parts are zero
    for at, c, v in [(1, 3, np.inf), (pos + 7, 9, -np.inf), (pos + 33, 3, np.inf)]:  # first page, inside the portion
        slot = tab[at // 64] * 64 + at % 64
        if where == "key":
            K[at, G - 1, 0, c] = v
            raw[slot, (G - 1) * maps * D + c] = 0x7f80 if v > 0 else 0xff80
        elif where == "value":
            V[at, 0, c] = v
            raw[slot, G * maps * D + c] = 0x7f80 if v > 0 else 0xff80
        elif at >= pos:
            q[at - pos, min(4, H - 1), 0, c] = v
    cache.upload(raw)
    vis = seen(pos, T, window, keep, 0)
    dist = np.maximum(np.arange(pos, pos + T)[:, None] - np.arange(pos + T)[None], 0)
    got = attend(gpu, kind, q, cache, table, pos0, T, pos, H, G, D, Dv, cap, window, keep, offsets=offsets)
    with np.errstate(invalid="ignore", over="ignore"):
        want = plain_heads(kind, q, K, V, vis, cap, offsets.astype(np.float64), dist)
    assert np.isfinite(want).any() and (np.isnan(got) == np.isnan(want)).all() and (got[np.isinf(want)] == want[np.isinf(want)]).all()
    ok = np.isfinite(want)
    assert np.isfinite(got[ok]).all() and rel(got[ok], want[ok]) < LIMIT
