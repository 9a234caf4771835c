"""Experts of a portion: the router's logits in tiles of tokens and experts are the bits of a logit by itself, the grouping kernel's lists for more slots
than its threads hold and more experts than it has threads, the weighted sum in whole pieces and number by number."""
import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, f32, from_dt, i32, release, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("T,E,W", [(2400, 4, 132), (301, 34, 64), (1025, 33, 512), (700, 32, 66)])
def test_logits_do_not_depend_on_the_tokens_of_a_call(gpu, dt, T, E, W):
    r, lib = np.random.default_rng(T), gpu.cuda_lib()
    h = dev(gpu, as_dt(dt, r.standard_normal((T, W)))[1])
    w, b = dev(gpu, f32(r.standard_normal((E, W)))), dev(gpu, f32(r.standard_normal(E)))
    z, idx, wt = zeros(gpu, T * E * 4), zeros(gpu, T * 2 * 4), zeros(gpu, T * 2 * 4)
    gpu.check(lib.ggb_op_moe_route(dt, h.ptr, W, T, w.ptr, b.ptr, E, 2, z.ptr, idx.ptr, wt.ptr))
    whole, es = z.download(np.uint32).reshape(T, E).copy(), 2 if dt == BF16 else 4
    for t in (0, 1, T // 2, T - 1):
        gpu.check(lib.ggb_op_moe_route(dt, h.ptr.value + t * W * es, W, 1, w.ptr, b.ptr, E, 2, z.ptr, idx.ptr, wt.ptr))
        assert np.array_equal(z.download(np.uint32, E), whole[t])


@pytest.mark.parametrize("n,top,E,identity", [(1, 1, 1, 0), (37, 2, 5, 1), (4096, 4, 32, 0), (8192, 2, 7, 3), (8193, 3, 40, 0), (30001, 1, 2050, 0), (64, 1, 1100, 100)])
def test_grouping(gpu, n, top, E, identity):
    r, lib = np.random.default_rng(n), gpu.cuda_lib()
    T = -(-n // top)
    n = T * top
    idx = i32(np.minimum(r.integers(0, E, n), r.integers(0, E, n)))
    ws = zeros(gpu, 4 * lib.ggb_moe_group_ints(n, E))
    gpu.check(lib.ggb_op_moe_group_identity(dev(gpu, idx).ptr, T, top, E, identity, ws.ptr))
    a = ws.download(np.int32)
    mt = lib.ggb_moe_max_tiles(n, E)
    offsets, rest = a[:E + 1], a[E + 1:]
    row_src, inv, te, tr, nt, row_expert = rest[:n], rest[n:2 * n], rest[2 * n:2 * n + mt], rest[2 * n + mt:2 * n + 2 * mt], rest[2 * n + 2 * mt], rest[2 * n + 2 * mt + 1:][:n]
    count = np.bincount(idx, minlength=E)
    assert np.array_equal(offsets, np.concatenate([[0], np.cumsum(count)]))
    assert np.array_equal(np.sort(inv), np.arange(n))
    assert np.array_equal(row_expert, np.repeat(np.arange(E), count)) and np.array_equal(row_expert[inv], idx)
    assert np.array_equal(row_src[inv], np.arange(n) // top)
    want = [(e, x) for e in range(E - identity) for x in range(offsets[e], offsets[e] + count[e], 64)]
    assert nt == len(want) and list(zip(te[:nt], tr[:nt])) == want


@pytest.mark.parametrize("W", [4, 30, 260, 2052])
@pytest.mark.parametrize("top", [1, 3, 6])
def test_weighted_sum(gpu, W, top):
    T, E = 9, 8
    r, lib = np.random.default_rng(W + top), gpu.cuda_lib()
    n = T * top
    ws = np.zeros(lib.ggb_moe_group_ints(n, E), np.int32)
    inv = r.permutation(n)
    ws[E + 1 + n:E + 1 + 2 * n] = inv
    y, wt, out = f32(r.standard_normal((n, W))), f32(r.random((T, top))), zeros(gpu, T * W * 4)
    gpu.check(lib.ggb_op_moe_combine(dev(gpu, y).ptr, dev(gpu, ws).ptr, dev(gpu, wt).ptr, T, top, E, W, out.ptr))
    want = (wt[:, :, None].astype(np.float64) * y[inv].reshape(T, top, W)).sum(1)
    assert np.abs(out.download(np.float32).reshape(T, W) - want).max() < top * 2.0 ** -23 * 8


@pytest.mark.parametrize("T,E", [(1203, 5), (2400, 5), (1203, 8), (2400, 8), (1203, 32), (2400, 32), (1184, 16), (1185, 16), (592, 32), (593, 32), (1183, 31), (1184, 30), (1185, 32), (1203, 20)])
def test_choice_does_not_depend_on_the_tokens_of_a_call(gpu, T, E):
    """up to 32 experts of a portion are chosen where their logits are computed: the bits of a token by itself, ties to the lower index"""
    W, top, r, lib = 132, 4, np.random.default_rng(E), gpu.cuda_lib()
    h = dev(gpu, as_dt(BF16, r.standard_normal((T, W)))[1])
    router = f32(r.standard_normal((E, W)))
    router[E - 1] = router[1]  # equal logits
    w, idx, wt = dev(gpu, router), zeros(gpu, T * top * 4), zeros(gpu, T * top * 4)
    z = zeros(gpu, T * E * 4)
    gpu.check(lib.ggb_op_moe_route(BF16, h.ptr, W, T, w.ptr, None, E, top, z.ptr, idx.ptr, wt.ptr))
    many = idx.download(np.int32).reshape(T, top).copy(), wt.download(np.uint32).reshape(T, top).copy()
    order = np.argsort(-z.download(np.float32).reshape(T, E), axis=1, kind="stable")[:, :top]
    assert np.array_equal(many[0], order)
    for t in (0, T // 2, T - 1):
        gpu.check(lib.ggb_op_moe_route(BF16, h.ptr.value + t * W * 2, W, 1, w.ptr, None, E, top, z.ptr, idx.ptr, wt.ptr))
        assert np.array_equal(idx.download(np.int32, top), many[0][t]) and np.array_equal(wt.download(np.uint32, top), many[1][t])


@pytest.mark.parametrize("T,W,E", [(150, 516, 64), (296, 512, 64), (297, 516, 64), (148, 512, 128), (150, 516, 128), (73, 1028, 256), (150, 508, 64), (300, 516, 40), (300, 514, 64)])
def test_logits_of_many_experts_are_the_bits_of_a_token_by_itself(gpu, T, W, E):
    top, r, lib = 3, np.random.default_rng(E + T), gpu.cuda_lib()
    for dt in (BF16, F32):
        h = dev(gpu, as_dt(dt, r.standard_normal((T, W)))[1])
        w, idx, wt = dev(gpu, f32(r.standard_normal((E, W)))), zeros(gpu, T * top * 4), zeros(gpu, T * top * 4)
        z, one = zeros(gpu, T * E * 4), zeros(gpu, E * 4)
        gpu.check(lib.ggb_op_moe_route(dt, h.ptr, W, T, w.ptr, None, E, top, z.ptr, idx.ptr, wt.ptr))
        many, got = z.download(np.float32).reshape(T, E), idx.download(np.int32).reshape(T, top).copy()
        assert np.array_equal(got, np.argsort(-many, axis=1, kind="stable")[:, :top])
        for t in (0, T // 2, T - 1):
            gpu.check(lib.ggb_op_moe_route(dt, h.ptr.value + t * W * (2 if dt == BF16 else 4), W, 1, w.ptr, None, E, top, one.ptr, idx.ptr, wt.ptr))
            assert np.array_equal(one.download(np.float32), many[t])


@pytest.mark.parametrize("T,E", [(3, 8), (1203, 8), (2400, 32), (3, 40), (1203, 40), (500, 32), (1100, 32), (1100, 16)])
def test_logits_that_are_no_numbers_choose_experts_that_exist(gpu, T, E):
    """tokens of NaN beside others, in the launch that computes the logits and in one of its own; the others' choice stays theirs"""
    W, top, r, lib = 132, 4, np.random.default_rng(E + T), gpu.cuda_lib()
    hv, hr = as_dt(BF16, r.standard_normal((T, W)))
    bad = [0, T // 2, T - 1]
    hr = hr.reshape(T, W).copy()
    hr[bad, 5] = 0x7fc0
    w, idx, wt, z = dev(gpu, f32(r.standard_normal((E, W)))), zeros(gpu, T * top * 4), zeros(gpu, T * top * 4), zeros(gpu, T * E * 4)
    gpu.check(lib.ggb_op_moe_route(BF16, dev(gpu, hr).ptr, W, T, w.ptr, None, E, top, z.ptr, idx.ptr, wt.ptr))
    got, logits = idx.download(np.int32).reshape(T, top), z.download(np.float32).reshape(T, E)
    assert ((got >= 0) & (got < E)).all() and np.isnan(logits[bad]).all()
    good = np.setdiff1d(np.arange(T), bad)
    assert np.array_equal(got[good], np.argsort(-logits[good], axis=1, kind="stable")[:, :top]) and np.isfinite(wt.download(np.float32).reshape(T, top)[good]).all()


@pytest.mark.parametrize("gather", [0, 1])
@pytest.mark.parametrize("counts,N,K", [([0, 1, 16, 17, 31, 33, 0, 160, 255, 0], 160, 448), ([256, 257, 0], 416, 64), ([513, 1, 2], 96, 192), ([700, 900], 1408, 128),
                                        ([3] * 300, 32, 64), ([17, 600, 0, 0], 288, 1024),
                                        # the same edges at sizes where the tiles are an expert's slots rather than rows
                                        ([0, 1, 16, 17, 31, 33, 0, 160, 255, 0], 416, 1024), ([0, 256, 257, 0, 1, 0, 0, 0], 288, 2048), ([0, 513, 1, 2] + [0] * 8, 160, 2048),
                                        ([700, 900] + [0] * 14, 288, 2048), ([3] * 300, 160, 256), ([3] * 300, 288, 64), ([3] * 200, 416, 192), ([17, 600, 0, 0, 5, 9, 30, 64], 288, 1024)])
def test_tiles_of_slots(gpu, counts, N, K, gather):
    """The grouped product at the edges of its tiles: halves of a tile without slots, groups without any, features that leave a CTA of a pair without work, fewer
    blocks of K than the ring has places.  Products are exact; a running sum is truncated once per 16 of K, at most 2^-23 of it."""
    r, lib = np.random.default_rng(len(counts) + N), gpu.cuda_lib()
    E, n = len(counts), sum(counts)
    assert n >= 512
    (w, wr), (a, ar) = as_dt(BF16, r.standard_normal((E, N, K))), as_dt(BF16, r.standard_normal((n, K)))
    idx = r.permutation(np.repeat(np.arange(E), counts))
    ws, c, y = zeros(gpu, 4 * lib.ggb_moe_group_ints(n, E)), zeros(gpu, n * N * 4), zeros(gpu, n * N * 2)
    gpu.check(lib.ggb_op_moe_group(dev(gpu, i32(idx)).ptr, n, 1, E, ws.ptr))
    lists = ws.download(np.int32)
    row_src, expert = lists[E + 1:E + 1 + n], np.repeat(np.arange(E), counts)
    dw, da = dev(gpu, wr), dev(gpu, ar)
    gpu.check(lib.ggb_op_moe_linear(BF16, dw.ptr, N, K, da.ptr, K, gather, n, 1, E, ws.ptr, 0, c.ptr, N))
    gpu.check(lib.ggb_op_moe_linear(BF16, dw.ptr, N, K, da.ptr, K, gather, n, 1, E, ws.ptr, 1, y.ptr, N))  # the square of what is positive
    rows = a[row_src] if gather else a
    want = np.empty((n, N))
    for e in range(E):
        want[expert == e] = rows[expert == e] @ w[e].T
    got = c.download(np.float32).reshape(n, N)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < (K / 16 + 8) * 2.0 ** -23 + 1e-7
    square = from_dt(BF16, y, (n, N))
    assert np.array_equal(square, as_dt(BF16, np.maximum(got, np.float32(0)) ** 2)[0])


@pytest.mark.parametrize("E", [8192, 8193, 9001])
def test_more_groups_than_are_listed(gpu, E):
    """lists that a program has made itself, of more experts than the slots' kernel has room for"""
    r, lib, N, K, n = np.random.default_rng(E), gpu.cuda_lib(), 32, 64, 700
    idx = r.permutation(np.concatenate([r.integers(0, E, n - 70), np.full(67, 4000), [0, E - 1, E - 1]]))
    order = np.argsort(idx, kind="stable")
    lists = np.zeros(int(lib.ggb_moe_group_ints(n, E)), dtype=np.int32)
    lists[:E + 1] = np.concatenate([[0], np.cumsum(np.bincount(idx, minlength=E))])
    lists[E + 1:E + 1 + n] = order
    (w, wr), (a, ar) = as_dt(BF16, r.standard_normal((E, N, K))), as_dt(BF16, r.standard_normal((n, K)))
    ws, dw, da, c = dev(gpu, lists), dev(gpu, wr), dev(gpu, ar), zeros(gpu, n * N * 4)
    want = np.einsum("nk,nfk->nf", a[order], w[idx[order]])
    for gather in (1, 0):
        rows = da if gather else dev(gpu, ar[order])
        gpu.check(lib.ggb_op_moe_linear(BF16, dw.ptr, N, K, rows.ptr, K, gather, n, 1, E, ws.ptr, 0, c.ptr, N), "moe_linear")
        got = c.download(np.float32).reshape(n, N)
        assert np.linalg.norm(got - want) / np.linalg.norm(want) < (K / 16 + 8) * 2.0 ** -23 + 1e-7
