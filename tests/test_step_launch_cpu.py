"""Kernels that are launched before the one ahead of them has ended: every one of them waits (step_wait) before it touches memory, and no
pointer parameter promises the compiler that its memory is not written meanwhile (__restrict__), which would let it read early."""
import glob
import os
import re

import gemma_ggml_b200 as G

CSRC = os.path.join(os.path.dirname(G.CUDA_LIB), "csrc")


def kernels():
    """(file, name) -> (parameter list, body) of every __global__ function"""
    out = {}
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__", s):
            i = s.index("{", m.start())
            depth, k = 0, i
            while True:
                depth += {"{": 1, "}": -1}.get(s[k], 0)
                if depth == 0:
                    break
                k += 1
            sig = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", s[m.start():i])
            name = re.search(r"(\w+)\s*\(", sig).group(1)
            out[path, name] = (sig, s[i + 1:k])
    return out


def launched():
    names = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        s = open(path).read()
        for m in re.finditer(r"ggb_launch_step\(\s*(\w+)", s):
            name = m.group(1)
            if name == "k":  # a variable
                name = re.findall(r"auto k = (\w+)", s[:m.start()])[-1]
            names.add((path, name))
    return names


def test_every_early_launched_kernel_waits_before_it_touches_memory():
    ks, names = kernels(), launched()
    waiting = {n for n, (_, body) in ks.items() if "step_wait()" in body}
    assert len(names) > 15 and names == waiting
    for n in names:
        ahead = re.sub(r"(extern )?__shared__[^;]*;", "", ks[n][1].split("step_wait()")[0])
        assert not re.search(r"\[|->|[=(,]\s*\*\s*\w|\b(if|return|for|while)\b", ahead), (n, ahead)


def test_no_pointer_of_theirs_is_restrict():
    ks = kernels()
    assert not [n for n in launched() if "__restrict__" in ks[n][0]]


def test_a_kernel_whose_wait_ran_out_lets_its_copies_arrive():
    """Behind a wait that gave up, copies that were requested are still under way: no more are requested, and the CTA outlives them."""
    waiting = {n: body for n, (_, body) in kernels().items() if "mbar_wait_bounded(" in body}
    assert len(waiting) >= 5
    for n, body in waiting.items():
        end = body[body.rindex("settle(dead);"):]
        assert "tmem_free512" in end, n
        for m in re.finditer(r"mbar_expect_tx\(", body):
            ahead = body[:m.start()]
            since = ahead[ahead.rindex("mbar_wait_bounded("):]
            assert re.search(r"if \(!$", ahead[:ahead.rindex("mbar_wait_bounded(")]) and "break;" in since or re.search(r"if \($", ahead[:ahead.rindex("mbar_wait_bounded(")]), n


def test_a_copying_warp_whose_wait_ran_out_leaves_every_loop():
    """Copies by the threads (cp.async) behind a wait by whole warps: where the place that they copy from is carried from one tile to the next, a wait that gave up
    ends the loop over tiles, too: the place is no place of the following tile."""
    found = 0
    for n, (_, body) in kernels().items():
        for m in re.finditer(r"for \(([^;]*);([^;]*); [^()]*\b(\w+) -= [^()]*\) \{", body):  # a loop that carries a position
            depth, k = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(body[k], 0)
                k += 1
            loop = body[m.end():k]
            if "mbar_wait_warp(" not in loop or "cp_async16(" not in loop:
                continue
            found += 1
            flags = re.findall(r"if \(!\((\w+) = mbar_wait_warp\(", loop)
            assert loop.count("mbar_wait_warp(") == len(flags) and all(re.search(r"\b%s\b" % f, m.group(2)) for f in flags), n
    assert found >= 1


def test_barriers_of_a_cluster_hold_for_a_warp_whose_lanes_are_apart():
    """Lanes that leave a wait each by its own answer may still be apart where the roles of a kernel end: a cluster's barrier that such a warp came to in parts would count
    it twice.  Every one is behind a vote, in the form that does not take the lanes for together."""
    found = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        s = re.sub(r"//[^\n]*", "", open(path).read())
        assert not re.search(r"barrier\.cluster\.[a-z.]*aligned", s), path
        for m in re.finditer(r"barrier\.cluster\.arrive", s):
            found += 1
            assert re.search(r"warp_meet\(\);\s*asm volatile\(\"$", s[:m.start()]), path
    assert found == 1  # cluster_arrive, which everything else calls
    # and tensor memory is given back by whole warps, the ones that issued MMAs among them
    s = open(os.path.join(CSRC, "tc.cuh")).read()
    assert len(re.findall(r"warp_meet\(\);\s*asm volatile\(\"tcgen05\.dealloc", s)) == len(re.findall(r"tcgen05\.dealloc", s)) == 2


def test_a_pair_of_ctas_outlives_what_is_sent_to_either():
    """The products by pairs of CTAs: whoever fills stages, and whoever issues MMAs, waits at its end for the arrivals that nobody else waits for, and neither CTA leaves
    before both have given their tensor memory back."""
    ks = {n: body for n, (_, body) in kernels().items() if n[0].endswith("gemm.cu") and "umma_arrive_pair(" in body}
    assert len(ks) == 2
    for n, body in ks.items():
        end = body[body.rindex("tmem_free512_pair"):]
        assert "cluster_sync();" in end and re.search(r"warp_meet\(\);\s*__syncthreads\(\);\s*if \(warp == 2\) settle\(dead\);\s*cluster_sync\(\);", body), n
        fills, issues = body.index("warp == 0) {"), body.index("} else if (warp == 1 && rank == 0) {")
        assert re.search(r"for \(int k = 0; k < kS\w+ && mbar_wait_bounded\(bars \+ EMPTY", body[fills:issues]), n
        after = body[body.index("umma_arrive_pair(bars + ACC_FULL", issues):]
        assert "mbar_wait_bounded(bars + ACC_FREE" in after[:after.index("} else if")], n
