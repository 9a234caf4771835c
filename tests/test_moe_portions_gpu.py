"""Experts of a portion: the router's logits in tiles of tokens and experts are the bits of a logit by itself, the grouping kernel's lists for more slots
than its threads hold and more experts than it has threads, the weighted sum in whole pieces and number by number."""
import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, f32, i32, release, zeros

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
