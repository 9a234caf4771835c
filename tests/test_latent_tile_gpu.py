"""The tensor-core form of latent attention over portions (csrc/latent_tile.cuh) against float64, at the edges of its tiles: 128 rows
(tokens x heads), 256 positions, blocks of 64 coordinates and latents cut in two above 256.  The tensor cores truncate a running fp32 sum
once per 16 products, as in every product of the library: a score is off by at most 3 QK / 16 steps of 2^-23 of the largest one, and the
weights, sums and weighted sums by that factor (plus 3 n / 16 such steps of their own).  The output is rounded to bf16 (2^-9 at most)."""
import numpy as np
import pytest

from device_util import BF16, as_dt, dev, f32, from_dt, i32, release, zeros

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# H, R, Dr, Dv, T, pos, window, splits, page, gate, scale
CASES = [(16, 512, 64, 128, 33, 250, 0, 1, 64, 0, 1.0), (16, 512, 64, 128, 32, 224, 100, 2, 64, 1, 3.0), (8, 256, 32, 64, 40, 0, 0, 1, 7, 0, 1.0), (4, 128, 64, 16, 65, 700, 300, 3, 64, 1, 0.5),
         (1, 32, 16, 16, 129, 127, 0, 1, 64, 0, 1.0), (3, 96, 0, 48, 50, 1, 1, 2, 16, 0, 2.0), (128, 64, 16, 32, 9, 255, 0, 2, 64, 0, 1.0), (5, 320, 48, 256, 100, 513, 0, 7, 64, 0, 8.0),
         (16, 480, 32, 80, 200, 56, 256, 1, 64, 1, 1.0), (7, 288, 16, 96, 31, 0, 0, 4, 64, 0, 1.0),
         # unsplit positions: up to two CTAs' rows on the CUDA cores, more here
         (1, 32, 16, 16, 256, 2, 0, 1, 64, 0, 1.0), (1, 32, 16, 16, 257, 2, 0, 1, 64, 0, 1.0), (16, 512, 64, 128, 16, 40, 0, 1, 64, 0, 1.0), (16, 512, 64, 128, 17, 40, 0, 1, 64, 0, 1.0)]


@pytest.mark.parametrize("H,R,Dr,Dv,T,pos,window,ns,page,gate,scale", CASES)
def test_parts_and_output(gpu, H, R, Dr, Dv, T, pos, window, ns, page, gate, scale):
    r = np.random.default_rng(R + T)
    lib, QK, n = gpu.cuda_lib(), R + Dr, pos + T
    ld, pages = int(lib.ggb_latent_cache_ld(R, Dr)), (n + page - 1) // page
    table = r.permutation(pages + 2)[:pages].astype(np.int32)
    cache, raw = as_dt(BF16, r.standard_normal(((pages + 2) * page, ld)))
    rows = cache[table[np.arange(n) // page].astype(np.int64) * page + np.arange(n) % page][:, :QK]
    qa, (w, wraw) = f32(r.standard_normal((T, H, QK)) * scale * QK ** -0.5), as_dt(BF16, r.standard_normal((H, Dv, R)) * R ** -0.5)
    sink, g = f32(r.standard_normal(H)), f32(r.standard_normal((T, H)))
    part, out = zeros(gpu, lib.ggb_latent_attn_scratch_bytes(T, H, R, ns)), zeros(gpu, T * H * Dv * 2)
    gpu.check(lib.ggb_op_latent_attn_window(BF16, dev(gpu, qa).ptr, dev(gpu, raw).ptr, dev(gpu, table).ptr, page, dev(gpu, i32([pos])).ptr, T, H, R, Dr, window, ns, part.ptr), "attn")
    gpu.check(lib.ggb_op_latent_attn_out_gated(BF16, part.ptr, ns, dev(gpu, sink).ptr, dev(gpu, wraw).ptr, T, H, R, Dv, dev(gpu, g).ptr if gate else None, H, out.ptr), "out")
    i, j = np.arange(pos, n)[:, None, None], np.arange(n)[None, None]
    s = np.einsum("thk,nk->thn", qa.astype(np.float64), rows)
    s = np.where((j <= i) & ((j > i - window) | (window <= 0)), s, -np.inf)
    m = s.max(2, keepdims=True)
    e = np.exp(s - m)
    got = part.download(np.float32, T * ns * H * (R + 2)).reshape(T, ns, H, R + 2).astype(np.float64)
    off = 3 * (QK / 16) * 2.0 ** -23 * np.abs(s[np.isfinite(s)]).max()
    assert np.abs(got[..., 0].max(1) - m[..., 0]).max() < off  # the parts hold the true maxima
    f = np.exp(got[..., 0] - m[:, None, :, 0])
    assert rel((got[..., 1] * f).sum(1), e.sum(2)) < off + 1e-6
    acc = np.einsum("thn,nr->thr", e, rows[:, :R])
    assert rel((got[..., 2:] * f[..., None]).sum(1), acc) < off + 3 * (n / 16) * 2.0 ** -23
    o = acc / (e.sum(2, keepdims=True) + np.exp(sink.astype(np.float64)[None, :, None] - m))
    want = np.einsum("thr,hvr->thv", o, w) * (1.0 / (1.0 + np.exp(-g.astype(np.float64)))[..., None] if gate else 1.0)
    assert rel(from_dt(BF16, out, (T, H, Dv)), want) < 2.5e-3


@pytest.mark.parametrize("where", ["rotated", "latent", "w_uv", "query", "nan"])
@pytest.mark.parametrize("H,R,Dr,Dv,T,pos,window,ns", [(5, 320, 48, 32, 40, 20, 0, 2), (4, 128, 16, 48, 33, 500, 300, 1), (4, 128, 16, 48, 70, 500, 300, 1)])
def test_infinities_as_plain_arithmetic_has_them(gpu, where, H, R, Dr, Dv, T, pos, window, ns):
    r = np.random.default_rng(R)
    lib, QK, n, page = gpu.cuda_lib(), R + Dr, pos + T, 64
    ld, pages = int(lib.ggb_latent_cache_ld(R, Dr)), (n + page - 1) // page
    table = r.permutation(pages).astype(np.int32)
    cache, raw = as_dt(BF16, r.standard_normal((pages * page, ld)))
    at = table[np.arange(n) // page].astype(np.int64) * page + np.arange(n) % page
    qa, (w, wraw) = f32(r.standard_normal((T, H, QK)) * QK ** -0.5), as_dt(BF16, r.standard_normal((H, Dv, R)) * R ** -0.5)
    bits = {np.inf: 0x7f80, -np.inf: 0xff80, np.nan: 0x7fc0}
    for j, c, v in [(pos - 1, R + 3, np.inf), (pos + 30, R + 3, -np.inf)] if where == "rotated" else [(pos + 30, 7, -np.inf)] if where == "latent" else [(pos + 20, 5, np.nan)] if where == "nan" else []:
        cache[at[j], c], raw[at[j], c] = v, bits[v]
    if where == "w_uv":
        w[1, 2, 9], wraw[1, 2, 9] = -np.inf, 0xff80
    if where == "query":
        qa[3, 2, R + 1] = np.inf
    part, out = zeros(gpu, lib.ggb_latent_attn_scratch_bytes(T, H, R, ns)), zeros(gpu, T * H * Dv * 2)
    gpu.check(lib.ggb_op_latent_attn_window(BF16, dev(gpu, qa).ptr, dev(gpu, raw).ptr, dev(gpu, table).ptr, page, dev(gpu, i32([pos])).ptr, T, H, R, Dr, window, ns, part.ptr), "attn")
    gpu.check(lib.ggb_op_latent_attn_out_gated(BF16, part.ptr, ns, None, dev(gpu, wraw).ptr, T, H, R, Dv, None, H, out.ptr), "out")
    want = np.empty((T, H, Dv))
    with np.errstate(invalid="ignore"):
        for t in range(T):
            rows = cache[at[max(0, pos + t - window + 1) if window else 0:pos + t + 1], :QK]
            for h in range(H):
                s = rows @ qa[t, h].astype(np.float64)
                p = np.exp(s - s.max())
                want[t, h] = w[h] @ ((p / p.sum()) @ rows[:, :R])
    got = from_dt(BF16, out, (T, H, Dv))
    assert np.isfinite(want).any() and not np.isfinite(want).all()
    assert (np.isnan(got) == np.isnan(want)).all() and (got[np.isinf(want)] == want[np.isinf(want)]).all()
    ok = np.isfinite(want)
    assert rel(got[ok], want[ok]) < 2.5e-3


def test_parts_on_any_4_byte_boundary(gpu):
    lib, T, H, R, Dr, Dv, pos, page = gpu.cuda_lib(), 40, 4, 64, 16, 32, 10, 64
    r = np.random.default_rng(2)
    ld = int(lib.ggb_latent_cache_ld(R, Dr))
    cache, table, p0 = dev(gpu, as_dt(BF16, r.standard_normal((page, ld)))[1]), dev(gpu, i32([0])), dev(gpu, i32([pos]))
    qa, w = dev(gpu, f32(r.standard_normal((T, H, R + Dr)) * 0.1)), dev(gpu, as_dt(BF16, r.standard_normal((H, Dv, R)) * R ** -0.5)[1])
    n, got = int(lib.ggb_latent_attn_scratch_bytes(T, H, R, 1)), []
    for skip in (0, 1):
        part, out = zeros(gpu, n + 16), zeros(gpu, T * H * Dv * 2)
        gpu.check(lib.ggb_op_latent_attn(BF16, qa.ptr, cache.ptr, table.ptr, page, p0.ptr, T, H, R, Dr, 1, part.ptr.value + 4 * skip), "attn")
        gpu.check(lib.ggb_op_latent_attn_out_gated(BF16, part.ptr.value + 4 * skip, 1, None, w.ptr, T, H, R, Dv, None, H, out.ptr), "out")
        got.append(from_dt(BF16, out, (T, H, Dv)))
    assert np.abs(got[0]).max() > 0.1 and rel(got[1], got[0]) < 3e-3  # two forms of the output product: a rounding to bf16


@pytest.mark.parametrize("T", [8, 64])
def test_latents_too_wide_for_the_output_product_are_refused_for_every_portion(gpu, T):
    lib, H, R, Dv = gpu.cuda_lib(), 2, 2048, 16
    part, w, out = zeros(gpu, T * H * (R + 2) * 4), zeros(gpu, H * Dv * R * 2), zeros(gpu, T * H * Dv * 2)
    assert lib.ggb_op_latent_attn_out_gated(BF16, part.ptr, 1, None, w.ptr, T, H, R, Dv, None, H, out.ptr) != 0
