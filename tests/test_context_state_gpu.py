"""What the library keeps between calls belongs to its context: ggb_shutdown gives the memory back, and after another ggb_init every form of the
products runs as before.  A captured product finds the workspace of an earlier one of its T and N, and keeps it when a larger one takes its place.
Each in a process of its own.  And a wait
that ran out in a kernel is reported once, by the call that next waits for the GPU."""
import ctypes as C
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# the host-mapped word a kernel sets
FLAG = "_Z19ggb_wait_error_flagv"

SHUTDOWN = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np, torch
import gemma_ggml_b200 as G
from device_util import BF16, as_dt, dev, release, zeros

def products():
    lib, out = G.cuda_lib(), []
    for T, N, K in [(1024, 2048, 8192), (64, 2048, 8192), (128, 256, 1024)]:
        r = np.random.default_rng(N)
        w, a, c = dev(G, as_dt(BF16, r.standard_normal((N, K)))[1]), dev(G, as_dt(BF16, r.standard_normal((T, K)))[1]), zeros(G, T * N * 4)
        G.check(lib.ggb_op_linear(BF16, w.ptr, N, K, a.ptr, K, T, c.ptr, N), "linear")
        out.append(c.download(np.float32))
    del w, a, c
    release()
    return out

G.init(0)
first = products()
G.sync()
held = torch.cuda.mem_get_info(0)[0]
G.check(G.cuda_lib().ggb_shutdown())
freed = torch.cuda.mem_get_info(0)[0] - held
assert freed >= 1 << 24, freed  # the sums of a product cut along K: 2 x 1024 x 2048 numbers
G.check(G.cuda_lib().ggb_init(0))
for x, y in zip(first, products()):
    assert (x == y).all()
G.cuda_lib()._Z19ggb_wait_error_flagv.restype = C.POINTER(C.c_int)
G.cuda_lib()._Z19ggb_wait_error_flagv()[0] = 1
assert G.cuda_lib().ggb_shutdown() != 0
print("ok")
"""


CAPTURE = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np
import gemma_ggml_b200 as G
from device_util import BF16, as_dt, dev, zeros

G.init(0)
lib, T, N, K = G.cuda_lib(), 192, 2048, 8192
r = np.random.default_rng(1)
(w, wr), (a, ar) = as_dt(BF16, r.standard_normal((N, K))), as_dt(BF16, r.standard_normal((T, K)))
dw, da, c, c2 = dev(G, wr), dev(G, ar), zeros(G, T * N * 4), zeros(G, T * N * 4)
G.check(lib.ggb_op_linear(BF16, dw.ptr, N, 128, da.ptr, 128, T, c.ptr, N), "linear")  # too short to be cut along K
G.sync()
G.check(lib.ggb_capture_begin())
rc = lib.ggb_op_linear(BF16, dw.ptr, N, K, da.ptr, K, T, c.ptr, N)
g = C.c_void_p()
G.check(lib.ggb_capture_end(C.byref(g)))
G.check(rc, "captured linear")
G.check(lib.ggb_graph_launch(g))
G.check(lib.ggb_op_linear(BF16, dw.ptr, N, K, da.ptr, K, T, c2.ptr, N), "linear")
got, again, want = c.download(np.float32).reshape(T, N), c2.download(np.float32).reshape(T, N), a @ w.T
assert (got == again).all() and np.linalg.norm(got - want) < 1e-4 * np.linalg.norm(want)
print("ok")
"""

# graphs of a product cut along K and of a gathered product of experts, behind larger ones that take their workspaces' place
GROWN = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np
import gemma_ggml_b200 as G
from device_util import BF16, as_dt, dev, zeros
from test_moe_few_slots_gpu import Portion

G.init(0)
lib, N, K = G.cuda_lib(), 256, 4096
r = np.random.default_rng(1)
dw, da, c, c2 = dev(G, as_dt(BF16, r.standard_normal((N, K)))[1]), dev(G, as_dt(BF16, r.standard_normal((1024, K)))[1]), zeros(G, 64 * N * 4), zeros(G, 1024 * N * 4)
p, big = Portion(G, 150, 4, 8, 64, 256), Portion(G, 2048, 4, 8, 64, 1024, seed=2)
def small():
    return lib.ggb_op_linear(BF16, dw.ptr, N, K, da.ptr, K, 64, c.ptr, N) or p.launch()
G.check(small())
first = c.download(np.float32), p.c.download(np.float32)
G.check(lib.ggb_capture_begin())
rc = big.launch()
g = C.c_void_p()
lib.ggb_capture_end(C.byref(g))
assert rc != 0  # no room, and none can be had there
graphs = []
for _ in range(2):
    G.check(lib.ggb_capture_begin())
    rc = small()
    g = C.c_void_p()
    G.check(lib.ggb_capture_end(C.byref(g)))
    G.check(rc)
    graphs.append(g)
    G.check(lib.ggb_op_linear(BF16, dw.ptr, N, K, da.ptr, K, 1024, c2.ptr, N))
    G.check(big.launch())
    G.sync()
    for g in graphs:
        c.zero(); p.c.zero()
        G.check(lib.ggb_graph_launch(g))
        assert (c.download(np.float32) == first[0]).all() and (p.c.download(np.float32) == first[1]).all()
G.check(lib.ggb_shutdown())
print("ok")
"""

# a gathered product of experts captured ahead of any other: no workspace for copied rows, none needed; outside, copied rows are the faster form
FIRST = """
import sys
sys.path[:0] = sys.argv[1:3]
import ctypes as C
import numpy as np
import gemma_ggml_b200 as G
from test_moe_few_slots_gpu import Portion

G.init(0)
lib, p = G.cuda_lib(), Portion(G, 150, 4, 8, 64, 256)
G.check(lib.ggb_capture_begin())
rc = p.launch()
g = C.c_void_p()
G.check(lib.ggb_capture_end(C.byref(g)))
G.check(rc)
G.check(lib.ggb_graph_launch(g))
got, want = p.c.download(np.float32).reshape(-1, 64), p.want()[1]
p.c.zero()
G.check(p.launch())
again = p.c.download(np.float32).reshape(-1, 64)
for y in (got, again):
    assert np.linalg.norm(y - want) / np.linalg.norm(want) < (256 / 16 + 8) * 2.0 ** -23 + 1e-7
print("ok")
"""


@pytest.mark.parametrize("program", [SHUTDOWN, CAPTURE, GROWN, FIRST], ids=["shutdown", "capture", "grown", "first"])
def test_in_a_process_of_its_own(program):
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", program, os.path.dirname(tests), tests], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_a_wait_that_ran_out_is_an_error_once(gpu):
    lib, flag = gpu.cuda_lib(), getattr(gpu.cuda_lib(), FLAG)
    flag.restype = C.POINTER(C.c_int)
    word, host = flag(), (C.c_char * 16)()
    buf = gpu.DeviceBuffer(16)
    for call in (lambda: lib.ggb_sync(), lambda: lib.ggb_download(host, buf.ptr, 16)):
        assert call() == 0
        word[0] = 1
        assert call() != 0 and b"wait ran out" in lib.ggb_last_error()
        assert call() == 0 and word[0] == 0
