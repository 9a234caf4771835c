"""Recurrences of a portion, eight tokens at a time (csrc/recurrent.cu), against the same operator fed token by token (which is held to float64 in
test_begupel_ops_gpu.py and test_kibilix_ops_gpu.py): chunks left over, key and value sizes between the padded ones, more heads to a key head than a preparing
CTA has warps; portions cut at whole chunks and portions longer than the workspace are the same bits.  Both forms are fp32 multiply-adds over the same
terms in another order: a few 2^-24 per token of memory."""
import os
import subprocess
import sys

import numpy as np
import pytest

from device_util import dev, f32, release, zeros

pytestmark = pytest.mark.gpu
RULES = ["head", "channel", "decays", "lightning"]


@pytest.fixture(autouse=True)
def _release_buffers():
    yield
    release()


class Portion:
    def __init__(self, gpu, rule, T, H, G, D, Dv):
        r = np.random.default_rng(T + D + H)
        self.gpu, self.rule, self.T, self.H, self.G, self.D, self.Dv = gpu, rule, T, H, H if rule == "lightning" else G, D, Dv
        self.ld = 2 * self.G * D + H * Dv + 3
        self.na = H if rule == "head" else H * D
        x, a = r.standard_normal((T, self.ld)), r.standard_normal((T, self.na))
        if rule == "decays":
            a = r.uniform(0.2, 1.0, a.shape)
        self.x, self.a, self.b = dev(gpu, f32(x)), dev(gpu, f32(a)), dev(gpu, f32(r.standard_normal((T, H))))
        self.A_log, self.bias = dev(gpu, f32(r.uniform(-1.0, 1.0, H))), dev(gpu, f32(r.uniform(-4.0, 0.0, self.na)))
        self.decay, self.s0 = dev(gpu, f32(np.concatenate([[1.0], r.uniform(0.3, 0.999, H - 1)]))), f32(r.standard_normal((H, D, Dv)) * 0.1)

    def run(self, cuts):
        lib, st, o = self.gpu.cuda_lib(), dev(self.gpu, self.s0), zeros(self.gpu, self.T * self.H * self.Dv * 4)
        H, G, D, Dv, t = self.H, self.G, self.D, self.Dv, 0
        for n in cuts:
            q = self.x.ptr.value + 4 * t * self.ld
            k, v, out, a, b = q + 4 * G * D, q + 8 * G * D, o.ptr.value + 4 * t * H * Dv, self.a.ptr.value + 4 * t * self.na, self.b.ptr.value + 4 * t * H
            if self.rule == "head":
                rc = lib.ggb_op_gated_delta(q, k, v, self.ld, b, a, H, n, H, G, D, Dv, self.A_log.ptr, self.bias.ptr, st.ptr, out, H * Dv)
            elif self.rule == "lightning":
                rc = lib.ggb_op_lightning_attn(q, k, v, self.ld, n, H, D, Dv, self.decay.ptr, st.ptr, out, H * Dv)
            else:
                given = self.rule == "decays"
                rc = lib.ggb_op_channel_delta(q, k, v, self.ld, b, H, a, H * D, int(given), n, H, G, D, Dv, None if given else self.A_log.ptr, None if given else self.bias.ptr,
                                              st.ptr, out, H * Dv)
            self.gpu.check(rc)
            t += n
        assert t == self.T
        return o.download(np.float32).reshape(self.T, -1), st.download(np.float32)


def rel(a, b):
    return np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64))


@pytest.mark.parametrize("rule", RULES)
@pytest.mark.parametrize("T,H,kv,D,Dv", [(16, 4, 2, 64, 64), (17, 2, 1, 12, 5), (31, 9, 1, 65, 16), (75, 3, 3, 128, 17), (40, 4, 4, 130, 40), (24, 2, 2, 256, 33), (50, 20, 2, 33, 64)])
def test_chunks_against_single_tokens(gpu, rule, T, H, kv, D, Dv):
    p = Portion(gpu, rule, T, H, kv, D, Dv)
    (o, s), (o1, s1) = p.run([T]), p.run([1] * T)
    assert rel(o, o1) < 2e-6 and rel(s, s1) < 2e-6


@pytest.mark.parametrize("rule", RULES)
def test_cuts_at_whole_chunks_change_nothing(gpu, rule):
    # 24 heads of 256 x 256: a chunk takes up to 830 KB of the workspace, so that the whole is several segments
    p = Portion(gpu, rule, 700, 24, 24, 256, 256)
    (o, s), (o1, s1) = p.run([700]), p.run([168, 400, 132])
    assert np.array_equal(o, o1) and np.array_equal(s, s1)


CAPTURE = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np
import gemma_ggml_b200 as G
from test_recurrence_chunks_gpu import Portion, rel
from device_util import dev, zeros

G.init(0)
lib, p = G.cuda_lib(), Portion(G, "head", 40, 4, 2, 64, 64)
st, o = dev(G, p.s0), zeros(G, 40 * 4 * 64 * 4)
G.sync()
G.check(lib.ggb_capture_begin())
q = p.x.ptr.value
rc = lib.ggb_op_gated_delta(q, q + 4 * 128, q + 8 * 128, p.ld, p.b.ptr, p.a.ptr, 4, 40, 4, 2, 64, 64, p.A_log.ptr, p.bias.ptr, st.ptr, o.ptr, 256)
g = C.c_void_p()
G.check(lib.ggb_capture_end(C.byref(g)))
G.check(rc, "captured portion")
G.check(lib.ggb_graph_launch(g))
want, state = p.run([40])
assert rel(o.download(np.float32).reshape(40, -1), want) < 2e-6 and rel(st.download(np.float32), state) < 2e-6
print("ok")
"""


def test_a_first_portion_inside_a_capture():
    """The workspace does not exist yet and cannot be had: the token by token form is captured."""
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", CAPTURE, os.path.dirname(tests), tests], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
