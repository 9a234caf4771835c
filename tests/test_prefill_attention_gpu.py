"""Attention of a prompt on the tensor cores (csrc/prefill_attention.cu) at the edges of its tiles: query rows and keys left over, groups of 1 to 8 heads
and one that does not divide the rows, portions behind a filled cache, and numbers that are not finite.  Against float64 on the same fp16 numbers: every
weight is rounded to fp16 once (2^-11), and weights are positive, so an output is off by at most 2^-11 of the sum of |weight * value|."""
import numpy as np
import pytest

from device_util import dev, f32, release, zeros
from safolorn_fixture import bf16_round

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def run(gpu, q, k, v, pos0):
    T, H, D = q.shape
    o, ob = zeros(gpu, T * H * D * 4), zeros(gpu, T * H * D * 2)
    gpu.check(gpu.cuda_lib().ggb_op_attn_prefill(dev(gpu, f32(q)).ptr, dev(gpu, k).ptr, dev(gpu, v).ptr, T, pos0, H, k.shape[1], D, o.ptr, ob.ptr))
    return o.download(np.float32).reshape(T, H, D), ob.download(np.uint16).reshape(T, H, D)


def plain(q, k, v, pos0):
    """outputs and the sums of |weight * value|"""
    T, H, D = q.shape
    g = H // k.shape[1]
    out, size = np.zeros((T, H, D)), np.zeros((T, H, D))
    q16 = q.astype(np.float16).astype(np.float64)
    for h in range(H):
        K, V = k[:, h // g].astype(np.float64), v[:, h // g].astype(np.float64)
        for t in range(T):
            n = pos0 + t + 1
            s = K[:n] @ q16[t, h]
            p = np.exp(s - s.max())
            p /= p.sum()
            out[t, h], size[t, h] = p @ V[:n], p @ np.abs(V[:n])
    return out, size


@pytest.mark.parametrize("T,pos0,H,Hkv,D", [(16, 112, 8, 1, 256), (17, 111, 8, 1, 256), (130, 0, 8, 8, 64), (64, 0, 4, 4, 128), (65, 63, 4, 1, 64), (33, 191, 6, 2, 192), (40, 1, 5, 1, 128),
                                            (16, 700, 4, 2, 256), (129, 300, 2, 2, 256),
                                            # key tiles dealt to 4, 8 and 2 CTAs, of which some have none
                                            (512, 0, 8, 1, 256), (200, 1000, 8, 1, 128), (300, 0, 8, 4, 64)])
def test_prompts(gpu, T, pos0, H, Hkv, D):
    r = np.random.default_rng(T + pos0 + H)
    q = r.standard_normal((T, H, D)) * 2.0 * D ** -0.5
    k, v = (r.standard_normal((pos0 + T, Hkv, D)).astype(np.float16) for _ in range(2))
    k[pos0 // 2] *= 4.0  # keys that stand out
    want, size = plain(f32(q), k, v, pos0)
    got, bf = run(gpu, q, k, v, pos0)
    assert (np.abs(got - want) <= 2.0 ** -10 * size + 1e-6).all()
    assert np.array_equal(bf, bf16_round(got)[1])


def test_numbers_that_are_not_finite(gpu):
    """An infinite value counts from the token on that sees it; a NaN in a query stays in its row."""
    T, H, Hkv, D = 100, 4, 2, 64
    r = np.random.default_rng(2)
    q = f32(r.standard_normal((T, H, D)) * D ** -0.5)
    k, v = (r.standard_normal((T, Hkv, D)).astype(np.float16) for _ in range(2))
    clean, _ = run(gpu, q, k, v, 0)
    v[40, 1, 3], q[7, 0, 5] = np.inf, np.nan
    got, _ = run(gpu, q, k, v, 0)
    assert np.isnan(got[7, 0]).all() and np.isinf(got[40:, 2:, 3]).all()
    rest = np.ones((T, H, D), bool)
    rest[7, 0] = False
    rest[40:, 2:, 3] = False
    assert (np.abs(got[rest] - clean[rest]) <= 2e-3).all()  # rows computed once more round every weight to fp16 behind its division


def test_the_switch_to_plain_kernels(gpu, monkeypatch):
    """GGB_PREFILL_ATTN_SIMPLE (and with it GGB_PREFILL_ATTN_GH4) picks the kernels without tensor cores for sizes that the tiles take, too."""
    r = np.random.default_rng(3)
    q = f32(r.standard_normal((130, 8, 128)) * 128 ** -0.5)
    k, v = (r.standard_normal((130, 1, 128)).astype(np.float16) for _ in range(2))
    want, size = plain(q, k, v, 0)
    tiles, _ = run(gpu, q, k, v, 0)
    monkeypatch.setenv("GGB_PREFILL_ATTN_SIMPLE", "1")
    simple, _ = run(gpu, q, k, v, 0)
    monkeypatch.setenv("GGB_PREFILL_ATTN_GH4", "1")
    four, _ = run(gpu, q, k, v, 0)
    for got in (simple, four):  # a weight's exponent and the weight are fp16 numbers
        assert (np.abs(got - want) <= 2.0 ** -7 * size).all() and not np.array_equal(got, tiles)
