"""Results that a kernel leaves in host memory beside the number of their call (mul_mat of host pointers)."""
import glob
import os
import re
import shutil
import subprocess

import pytest

import gemma_ggml_b200 as G

CSRC = os.path.join(os.path.dirname(G.CUDA_LIB), "csrc")


def test_a_word_for_another_processor_is_one_scalar_store():
    """Numbers that belong together, payload and tag, arrive together only where one scalar store of eight bytes writes them: the numbers of a vector store are
    stores of their own, in no stated order."""
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        for m in re.finditer(r'"(st\.[\w.:]*\bsys\b[\w.:]*)', open(path).read()):
            found += 1
            assert re.search(r"\.[bu]64$", m.group(1)) and not re.search(r"\.v[248]\b", m.group(1)), (path, m.group(1))
    assert found >= 2


PROGRAM = r"""
#include <assert.h>
#include <thread>
#include "host_words.cuh"
static uint64_t word(uint32_t call, float v) { uint32_t b; memcpy(&b, &v, 4); return (uint64_t)call << 32 | b; }
int main() {
    uint64_t mem[8] = {};
    host_words h;
    h.words = mem, h.n = 8;
    float y[8];
    auto never = [] { assert(0); return true; };
    // the first numbers are not zero, which is what a new word holds
    assert(h.next(never) && h.call == 1);
    for (int i = 0; i < 8; i++) mem[i] = word(1, 10.f + i); // a large call
    assert(h.take(y, 0, 8, [] { return 1; }) && y[0] == 10.f && y[7] == 17.f);
    // small calls until the numbers are used up: words 2 .. 7 keep the number 1
    h.call = UINT32_MAX - 1;
    assert(h.next(never) && h.call == UINT32_MAX);
    mem[0] = mem[1] = word(h.call, 3.f);
    assert(h.take(y, 0, 2, [] { return 1; }));
    // a kernel of an earlier call may still store: not this time, and the next one asks again
    assert(!h.next([] { return false; }) && !h.next([] { return false; }) && mem[7] >> 32 == 1);
    assert(h.next([] { return true; }) && h.call == 1);
    int asked = 0; // a large call of the same number: the old results are not its own
    assert(!h.take(y, 0, 8, [&] { asked++; return 0; }) && asked == 1);
    for (int i = 0; i < 7; i++) mem[i] = word(1, 20.f + i);
    assert(!h.take(y, 0, 8, [] { return -1; }));
    // a result that arrives between the look and the question, and one that takes long
    asked = 0;
    assert(h.take(y, 0, 8, [&] { if (++asked == 100000) mem[7] = word(1, 27.f); return asked < 100000 ? 1 : 0; }) && y[7] == 27.f && asked == 100000);
    assert(h.take(y + 1, 5, 1, [] { return -1; }) && y[1] == 25.f);
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="no C++ compiler")
def test_numbers_of_calls_that_begin_again_and_results_that_never_come(tmp_path):
    src, exe = tmp_path / "words.cpp", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)
