"""The packed K-quant mat-vec (csrc/kquants.cu: integer tensor-core tiles of 16 rows) at the edges of its tiles and rounds: a tile of one row, rows
left over, one super-block up to rounds of unequal super-blocks, several tiles a round; bit for bit against the scalar code."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


@pytest.mark.parametrize("wtype", [O.TYPE_Q4_K, O.TYPE_Q6_K])
@pytest.mark.parametrize("n,k,t", [(1, 256, 1), (15, 512, 2), (16, 768, 1), (17, 1024, 1), (130, 1280, 1), (31, 1792, 1), (33, 2304, 2), (5000, 256, 1), (47, 2560, 1),
                                   (18, 5120, 1), (9600, 2048, 1)])
def test_packed_tiles(gpu, wtype, n, k, t):
    rng, L = np.random.default_rng(n + k), gpu.cuda_lib()
    w = O.random_kquant_rows(rng, wtype, n, k)
    x = (rng.standard_normal((t, k)) * 1.5).astype(np.float32)
    act = O.quantize_q8_K(x)
    want = bits(O.mul_mat_blocks(wtype, w, act, k))
    q4 = wtype == O.TYPE_Q4_K
    wd, xd, ad = (gpu.DeviceBuffer.from_numpy(a) for a in (w, x, act))
    packed = gpu.DeviceBuffer(w.nbytes if q4 else L.ggb_q6k_packed_bytes(n, k))
    gpu.check((L.ggb_op_q4k_repack if q4 else L.ggb_op_q6k_repack)(wd.ptr, n, w.shape[1], k, packed.ptr))
    ld = n + 3
    dst = gpu.DeviceBuffer(4 * ld * t)
    for run in (lambda: L.ggb_op_mul_mat_kq_packed_f32(wtype, packed.ptr, n, k, xd.ptr, t, dst.ptr, ld),
                lambda: (L.ggb_op_mul_mat_q4k_packed if q4 else L.ggb_op_mul_mat_q6k_packed)(packed.ptr, n, k, ad.ptr, act.shape[1], t, dst.ptr, ld)):
        gpu.check(L.ggb_buffer_memset(dst.ptr, 0, 4 * ld * t))
        gpu.check(run())
        gpu.sync()
        got = dst.download(np.float32).reshape(t, ld)
        assert np.array_equal(bits(got[:, :n]), want) and not got[:, n:].any()
