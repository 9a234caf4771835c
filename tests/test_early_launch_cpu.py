"""Kernels that set themselves up ahead of their wait for the kernel before them (early_wait): nothing of theirs is __restrict__, a kernel with tensor
memory lets the next one in behind its allocation, and one whose copies may be under way outlives them."""
import glob
import os

import test_step_launch_cpu as steps


def early():
    return {n: v for n, v in steps.kernels().items() if "early_wait()" in v[1]}


def test_pointers_and_order():
    ks = early()
    assert len(ks) >= 8
    for n, (sig, body) in ks.items():
        assert "__restrict__" not in sig and "step_wait()" not in body, n
        if "tmem_alloc512" in body and "step_next()" in body:
            assert body.index("tmem_alloc512") < body.index("__syncthreads()") < body.index("step_next()"), n


def test_copies_of_a_kernel_without_tensor_memory():
    waiting = {n: body for n, (_, body) in steps.kernels().items() if "mbar_wait_lane(" in body}
    assert waiting
    for n, body in waiting.items():
        for part in body.split("mbar_expect_tx(")[:-1]:
            assert "break;" in part[part.rindex("if (!mbar_wait_lane("):], n
        assert "settle(dead);" in body[body.rindex("bulk_load("):], n


def test_every_launch_of_theirs_has_the_attribute():
    src = "".join(open(p).read() for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")))
    for _, name in early():
        assert name + "<<<" not in src, name
