"""Products on the tensor cores that ask nothing of sizes, strides and addresses (csrc/gemm_any.cu): fp32 matrices in three bf16 parts, bf16 matrices
of few rows or odd sizes; remainders of tiles and of K, pieces of K over a cluster, activations, numbers that are not finite.

A stage of 64 of K is a sum of 16-number products that the tensor cores truncate (four steps of the large terms, 2^-23 each at most; the smaller
parts' steps are 2^-8 of that); stages are added with rounding to nearest; fp32 leaves out products below 2^-24 of a term: 6e-7 in all."""
import numpy as np
import pytest

from device_util import BF16, F32, as_dt, dev, f32, from_dt, release, size_of, zeros

pytestmark = pytest.mark.gpu
TOL = 6e-7


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("T,N,K", [(9, 1, 129), (16, 127, 192), (17, 129, 200), (33, 1000, 333), (80, 256, 129), (81, 300, 1000), (160, 64, 4100), (63, 128, 8192), (500, 130, 257),
                                   (9, 5000, 640), (31, 2048, 2048)])
def test_products(gpu, dt, T, N, K):
    r = np.random.default_rng(T + N + K)
    wv, wr = as_dt(dt, r.standard_normal((N, K)) * K ** -0.5)
    lda, ldc = K + (K % 3), N + 5
    av, ar = as_dt(dt, r.standard_normal((T, lda)))
    av = av[:, :K]
    want, es = av @ wv.T, size_of(dt)
    for skip in (0, 1):  # rows that start on 16 bytes and rows that do not
        w, a = dev(gpu, np.concatenate([np.zeros(skip, wr.dtype), wr.ravel()])), dev(gpu, np.concatenate([np.zeros(skip, ar.dtype), ar.ravel()]))
        c = zeros(gpu, T * ldc * 4)
        gpu.check(gpu.cuda_lib().ggb_op_linear(dt, w.ptr.value + es * skip, N, K, a.ptr.value + es * skip, lda, T, c.ptr, ldc))
        got = c.download(np.float32).reshape(T, ldc)
        assert rel(got[:, :N], want) < TOL and not got[:, N:].any()


@pytest.mark.parametrize("dt", [BF16, F32])
@pytest.mark.parametrize("act", [1, 4])
def test_activations(gpu, dt, act):
    from math import erf
    T, N, K = 20, 300, 260
    r = np.random.default_rng(act)
    wv, wr = as_dt(dt, r.standard_normal((N, K)) * K ** -0.5)
    av, ar = as_dt(dt, r.standard_normal((T, K)))
    y = zeros(gpu, T * N * size_of(dt))
    gpu.check(gpu.cuda_lib().ggb_op_linear_act(dt, dev(gpu, wr).ptr, N, K, dev(gpu, ar).ptr, K, T, act, y.ptr))
    z = av @ wv.T
    want = np.maximum(z, 0.0) ** 2 if act == 1 else 0.5 * z * (1.0 + np.vectorize(erf)(z / np.sqrt(2.0)))
    assert rel(from_dt(dt, y, (T, N)), want) < (2.0 ** -8 if dt == BF16 else 2e-6)


def test_small_numbers_keep_their_bits(gpu):
    """fp32 numbers around 2^-110, 2^-120 and 2^-128, whose bf16 parts the smallest bf16 number would cut off, times large ones."""
    T, N, K = 40, 130, 300
    r = np.random.default_rng(8)
    w, a = f32(r.standard_normal((N, K))), f32(r.standard_normal((T, K)))
    c, out = zeros(gpu, T * N * 4), {}
    for e in (0, -110, -120, -128):
        ae, we = np.ldexp(a, e), np.ldexp(w, -e // 2)
        gpu.check(gpu.cuda_lib().ggb_op_linear(F32, dev(gpu, we).ptr, N, K, dev(gpu, ae).ptr, K, T, c.ptr, N))
        out[e] = c.download(np.float32).reshape(T, N)
        assert rel(out[e].astype(np.float64), ae.astype(np.float64) @ we.astype(np.float64).T) < TOL, e
    assert np.array_equal(np.ldexp(out[-110], 55), out[0])


@pytest.mark.parametrize("dt", [BF16, F32])
def test_numbers_that_are_not_finite(gpu, dt):
    """Infinities and NaN, and the largest numbers (which round up to an infinity in bf16), give what plain multiply-adds give."""
    T, N, K = 24, 140, 300
    r = np.random.default_rng(3)
    w, a = r.standard_normal((N, K)), r.standard_normal((T, K))
    w[3, 7], w[130, 299], w[9, 0], a[5, 250], a[23, 1] = np.inf, -np.inf, np.nan, np.inf, -np.inf
    w[20, 11] = a[7, 40] = 3.4e38  # times numbers of about 1e-3
    a[:, 11] *= 1e-3
    w[:, 40] *= 1e-3
    (wv, wr), (av, ar) = as_dt(dt, w), as_dt(dt, a)
    c = zeros(gpu, T * N * 4)
    gpu.check(gpu.cuda_lib().ggb_op_linear(dt, dev(gpu, wr).ptr, N, K, dev(gpu, ar).ptr, K, T, c.ptr, N))
    got = c.download(np.float32).reshape(T, N)
    with np.errstate(invalid="ignore", over="ignore"):
        want = (av[:, None, :] * wv[None]).sum(2).astype(np.float32)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isinf(got), np.isinf(want))
    assert np.array_equal(np.sign(got[np.isinf(want)]), np.sign(want[np.isinf(want)]))
    ok = np.isfinite(want)
    assert (np.abs(got[ok] - want[ok]) <= 1e-5 * np.abs(av[:, None, :] * wv[None]).sum(2)[ok] + 1e-6).all()


def test_a_portion_of_nan_takes_about_as_long(gpu):
    """Results that are not finite are computed once more together: a few times the time of finite ones (a thread a result was several hundred times)."""
    import time
    T, N, K = 333, 1408, 1000
    r = np.random.default_rng(4)
    w, a, lib = dev(gpu, f32(r.standard_normal((N, K)))), f32(r.standard_normal((T, K))), gpu.cuda_lib()
    c, took = zeros(gpu, T * N * 4), []
    for x in (a, np.full_like(a, np.nan)):
        d = dev(gpu, x)
        for n in (2, 20):
            gpu.sync()
            t = time.perf_counter()
            for _ in range(n):
                gpu.check(lib.ggb_op_linear(F32, w.ptr, N, K, d.ptr, K, T, c.ptr, N))
            gpu.sync()
        took.append(time.perf_counter() - t)
        assert np.isnan(c.download(np.float32)).all() == np.isnan(x).all()
    assert took[1] < 20 * took[0], took
    print("us: finite %.1f, NaN %.1f" % (took[0] / 20 * 1e6, took[1] / 20 * 1e6))
