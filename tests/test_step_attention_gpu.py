"""Attention of a step of few tokens (csrc/window_attention.cu, window_step_kernel): lanes that share a row in eights, sixteens and thirty-twos, tiles and
splits that end inside, kept first positions, one and two maps, both cache types; against float64 on the same cache."""
import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, f32, from_dt, i32, release, size_of, zeros

pytestmark = pytest.mark.gpu
PAGE = 16


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def plain(q, K, V, pos, window, keep, cap, lam):
    T, H, maps, D = q.shape
    G, out = K.shape[1], []
    for t in range(T):
        j = np.arange(pos + t + 1)
        j = j[(j < keep) | (j > pos + t - window)] if window else j
        row = []
        for h in range(H):
            g, o = h // (H // G), []
            for m in range(maps):
                s = K[j, g, m] @ q[t, h, m]
                if cap:
                    s = cap * np.tanh(s / cap)
                p = np.exp(s - s.max())
                o.append((p / p.sum()) @ V[j, g])
            row.append(o[0] if maps == 1 else (lambda x: x / np.sqrt((x ** 2).mean() + 1e-5) * 0.8)(o[0] - lam * o[1]))
        out.append(row)
    return np.array(out)


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("maps", [1, 2])
@pytest.mark.parametrize("D,Dv,H,kv", [(8, 8, 2, 1), (64, 64, 4, 2), (80, 64, 4, 1), (96, 128, 2, 2), (128, 128, 8, 2), (64, 128, 3, 3)])
@pytest.mark.parametrize("T,pos,window,keep", [(1, 0, 0, 0), (1, 31, 0, 0), (1, 700, 0, 0), (3, 40, 32, 4), (1, 299, 33, 50), (31, 5, 100, 0), (1, 2200, 0, 0)])
def test_steps(gpu, dt, maps, D, Dv, H, kv, T, pos, window, keep):
    G = kv
    r = np.random.default_rng(D + pos + T)
    n, ld = pos + T, (G * (maps * D + Dv) + 7) // 8 * 8
    pages = -(-n // PAGE)
    table = r.permutation(pages)
    cv, cr = as_dt(dt, r.standard_normal((pages * PAGE, ld)))
    rows = cv[table[np.arange(n) // PAGE] * PAGE + np.arange(n) % PAGE]
    K, V = rows[:, :G * maps * D].reshape(n, G, maps, D), rows[:, G * maps * D:G * (maps * D + Dv)].reshape(n, G, Dv)
    q = f32(r.standard_normal((T, H, maps, D)) * 1.5 * D ** -0.5)
    lib = gpu.cuda_lib()
    out, scratch = zeros(gpu, T * H * Dv * size_of(dt)), zeros(gpu, lib.ggb_window_attn_scratch_bytes(H * maps))
    args = (dt, dev(gpu, q).ptr, dev(gpu, cr).ptr, dev(gpu, i32(table)).ptr, PAGE, dev(gpu, i32([pos, 0, 0, 0])).ptr, T, H, G, D, Dv, window, keep, 30.0)
    if maps == 1:
        gpu.check(lib.ggb_op_masked_attn_gated(*args, None, None, 0, out.ptr, scratch.ptr))
    else:
        gpu.check(lib.ggb_op_diff_attn(*args, 0.35, 0.8, 1e-5, None, 0, out.ptr, scratch.ptr))
    got, want = from_dt(dt, out, (T, H, Dv)), plain(q.astype(np.float64), K, V, pos, window, keep, 30.0, float(np.float32(0.35)))
    # sums of up to 2200 fp32 terms; a difference of two maps divided by its root mean square magnifies their error a little
    tol = 2.0 ** -8 if dt == BF16 else 5e-6
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < tol


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("D,pos", [(64, 0), (64, 12), (128, 31), (128, 700), (256, 21)])
def test_infinite_values(gpu, dt, D, pos):
    """An infinite value at the newest position (which ends a tile that is not whole) and one at the first: infinities where they are, the rest as ever."""
    if dt == F32 and D == 256:
        D = 128
    r = np.random.default_rng(pos)
    n, H = pos + 1, 2
    c = r.standard_normal((-(-n // PAGE) * PAGE, 2 * D))
    c[n - 1, D + 3] = c[0, D + 6] = np.inf
    c[n - 1, D + 5] = -np.inf
    cv, cr = as_dt(dt, c)
    q = f32(r.standard_normal((1, H, D)) * D ** -0.5)
    lib = gpu.cuda_lib()
    out, scratch = zeros(gpu, H * D * size_of(dt)), zeros(gpu, lib.ggb_window_attn_scratch_bytes(H))
    gpu.check(lib.ggb_op_masked_attn_gated(dt, dev(gpu, q).ptr, dev(gpu, cr).ptr, dev(gpu, i32(np.arange(len(c) // PAGE))).ptr, PAGE, dev(gpu, i32([pos, 0, 0, 0])).ptr, 1, H, 1,
                                           D, D, 0, 0, 0.0, None, None, 0, out.ptr, scratch.ptr))
    got = from_dt(dt, out, (H, D))
    assert (got[:, [3, 6]] == np.inf).all() and (got[:, 5] == -np.inf).all()
    V = np.where(np.isinf(cv[:n, D:]), 0, cv[:n, D:])
    s = np.einsum("jd,hd->hj", cv[:n, :D], q[0].astype(np.float64))
    want = np.einsum("hj,jd->hd", np.exp(s - s.max(1, keepdims=True)) / np.exp(s - s.max(1, keepdims=True)).sum(1, keepdims=True), V)
    rest = [d for d in range(D) if d not in (3, 5, 6)]
    assert np.linalg.norm(got[:, rest] - want[:, rest]) / np.linalg.norm(want[:, rest]) < (2.0 ** -8 if dt == BF16 else 5e-6)
