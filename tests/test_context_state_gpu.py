"""What the library keeps between calls belongs to its context: ggb_shutdown gives the memory back, and after another ggb_init every form of the
products runs as before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import sys
sys.path[:0] = sys.argv[1:3]
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
print("ok")
"""


def test_shutdown_gives_the_workspaces_back():
    tests = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", PROGRAM, os.path.dirname(tests), tests], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
