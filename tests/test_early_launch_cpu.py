"""Kernels that set themselves up ahead of their wait for the kernel before them (early_wait): what they do ahead of it touches no memory but weights,
nothing of theirs is __restrict__, a kernel with tensor memory lets the next one in behind its allocation, and one whose copies may be under way
outlives them.  A kernel that does nothing ahead of its wait is a step kernel (test_step_launch_cpu)."""
import glob
import os
import re

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


def launched():
    """the kernels that ggb_launch_early launches; a variable stands for every kernel that its declaration and assignments name"""
    names = set()
    for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")):
        s = re.sub(r"//[^\n]*", "", open(p).read())
        for m in re.finditer(r"ggb_launch_early\(\s*(\w+)", s):
            if m.group(1) == "void":
                continue
            found = [m.group(1)]
            if not found[0].endswith("_kernel"):
                ahead = s[s.rindex("auto %s = " % found[0], 0, m.start()):m.start()]
                found = re.findall(r"\b(\w+_kernel)\b", "".join(re.findall(r"\b%s = ([^;]*);" % found[0], ahead)))
            assert found, (p, m.group())
            names |= {(p, n) for n in found}
    return names


def test_which_kernels_and_how():
    """Every kernel with an early_wait is launched by ggb_launch_early and every one that it launches has one; no other launch asks for the attribute."""
    ks = early()
    assert len(ks) >= 8 and launched() == set(ks)
    for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")):
        s = open(p).read()
        assert os.path.basename(p) in ("common.cuh", "decoder.cu") or "cudaLaunchKernelEx" not in s, p
        for _, name in ks:
            assert not re.search(name + r"(<[^;{}()]*>)?<<<", s), name


TOUCHES = r"->|\)\*\w|\w\s*\[|\*\s*reinterpret_cast|[=(,]\s*\*\s*\w|\b(__ldg|ldg?_stream_u4|load4|store4|tma_load\w*|bulk_load\w*|cp_async\w*|atomic\w*|memcpy)\("


def test_what_is_done_ahead_of_the_wait():
    ks, by_role = early(), set()
    for (p, name), (_, body) in ks.items():
        body = re.sub(r"(extern )?__shared__[^;]*;", "", body)
        at = body.index("early_wait()")
        if "if (is_a) early_wait()" not in body:  # every thread comes by
            assert len(enclosing(body, at)) == 0 and not re.search(TOUCHES, body[:at]), (name, re.search(TOUCHES, body[:at]))
            assert re.search(r"\*dead = 0;|s_dead = 0;", body[:at]), name
            continue
        # One lane comes by, ahead of the first copy of what the kernel before wrote.  The others: weights (their codes and scales) and, behind the wait
        # for the last MMA of a tile, which that copy feeds, results, residual and the operand of the next product
        by_role.add(name)
        assert at < min(m.start() for m in re.finditer(r"&maps\.a\b", body))
        assert all(m.group(1) in ("a", "w") for m in re.finditer(r"&maps\.(\w+)", body))
        done = [m.start() for m in re.finditer(r"mbar_wait_(?:warp|bounded)\(bars \+ (?:DONE|Q_ACC_FULL)\b", body)]
        for m in re.finditer(r"\b(load4|store4)\(|A\.geglu \+|A\.gelu\)", body):
            around = [text for _, text in enclosing(body, m.start())]
            assert any(d < m.start() and (enclosing(body, d) or [("", body)])[0][1] in around for d in done), (name, m.group())
        reads = re.findall(r"(?<!reinterpret_cast<)\*\s*reinterpret_cast<([^>]*)>\(([^;]*);", body)
        assert all("ctl + " in r or "gbase + " in r or "A.geglu + " in r for _, r in reads), (name, reads)
    assert by_role == {"gemm_quant_kernel", "gemm_quant_stream_kernel"}


# what they read by loads that take it for granted that nobody writes there while the kernel runs: rows of weight matrices and their scales
WEIGHTS = {"dense.cu": {"wr + k"}, "moe.cu": {"wr + k", "wu + k"},
           "kquants.cu": {"codes + (p * R + r) * 64 + 16 * (lane & 3)", "o + 128 * kTileRows + r * 64 + 16 * (lane & 3)", "reinterpret_cast<const uint4 *>(o + 16 * r)",
                          "reinterpret_cast<const uint4 *>(o + 192 * kTileRows + 16 * r)", "reinterpret_cast<const uint16_t *>(o + 208 * kTileRows + 2 * r)"},
           "prefill.cu": {"dp + 2 * (kb + G * u)", "reinterpret_cast<const __half2 *>(dp + 2 * fkb)"}}


def test_only_weights_by_read_only_loads():
    """What the kernel before writes is read by ordinary loads: a read-only one may be moved ahead of the wait, and may find what was there before."""
    seen = 0
    for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")):
        s, name = re.sub(r"//[^\n]*", "", open(p).read()), os.path.basename(p)
        if name == "common.cuh" or not re.search(r"\b(early|step)_wait\(\)", s):
            continue
        assert "global.nc" not in s, name
        for m in re.finditer(r"\b(__ldg|ldg_stream_u4)\(", s):
            depth, k = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(s[k], 0)
                k += 1
            assert s[m.end():k - 1] in WEIGHTS.get(name, ()), (name, s[m.end():k - 1])
            seen += 1
    assert seen >= 6


def enclosing(src, at):
    """(what stands ahead of it, its text) of every block around a place, the innermost first"""
    blocks, depth = [], 0
    for k in range(at - 1, -1, -1):
        depth += {"}": 1, "{": -1}.get(src[k], 0)
        if depth < 0:
            depth = 0
            end, open_ = k, 0
            while True:
                open_ += {"{": 1, "}": -1}.get(src[end], 0)
                if open_ == 0:
                    break
                end += 1
            blocks.append((src[max(src.rfind(c, 0, k) for c in ";{}") + 1:k], src[k:end]))
    return blocks


def test_who_waits():
    """A warp whose lanes leave a wait one by one may hand a buffer on that its last lanes still read or write.  So lanes wait for themselves only where one
    goes on: in a block of lane 0, or where a warp does nothing but issue MMAs, whose lanes meet in every election; any other warp waits by mbar_wait_warp."""
    alone = warps = 0
    one = re.compile(r"if \(lane == 0\)\s*$")
    for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")):
        if os.path.basename(p) == "tc.cuh":
            continue
        s = re.sub(r"//[^\n]*", "", open(p).read())
        for m in re.finditer(r"mbar_(wait_bounded|try|test)\(", s):
            alone += 1
            blocks = enclosing(s, m.start())
            role = next((text for _, text in blocks if "umma_" in text or "mma_block(" in text), "mbar_arrive(")
            assert any(one.search(h) for h, _ in blocks) or not re.search(r"mbar_arrive(_cluster)?\(|sts_u|st\.shared|lds_u|tmem_(load|store)", role), (p, s[m.start():m.start() + 80])
        for m in re.finditer(r"mbar_wait_warp\(", s):
            warps += 1
            assert not any(one.search(h) for h, _ in enclosing(s, m.start())), (p, s[m.start():m.start() + 80])
    assert alone > 20 and warps > 15


def test_copies_of_a_kernel_without_tensor_memory():
    waiting = {n: body for n, (_, body) in steps.kernels().items() if "mbar_wait_warp(" in body and "mbar_expect_tx(" in body and "tmem_alloc512" not in body}
    assert waiting
    for n, body in waiting.items():
        for part in body.split("mbar_expect_tx(")[:-1]:
            assert "break;" in part[part.rindex("if (!mbar_wait_warp("):], n
        assert "settle(dead);" in body[body.rindex("bulk_load("):], n


def test_clusters_with_tensor_memory():
    """Their CTAs ask for so much shared memory that an SM has room for one: two clusters never hold what the other one waits for."""
    seen = 0
    for p in glob.glob(os.path.join(steps.CSRC, "*.cu*")):
        s = re.sub(r"//[^\n]*", "", open(p).read())
        for m in re.finditer(r"ggb_launch_early\(\s*\w+, ggb_cluster\{([^}]*)\},", s):
            if "tmem_alloc512" not in s or m.group(1) == "1, 1, 1":
                continue
            args, depth, last, k = [], 0, m.end(), m.end()
            while depth >= 0:  # grid, block, shared memory, the kernel's own
                depth += {"(": 1, ")": -1, "{": 1, "}": -1}.get(s[k], 0)
                if s[k] == "," and not depth:
                    args.append(s[last:k].strip())
                    last = k + 1
                k += 1
            smem = args[2]
            assert re.search(r"%s >= kOneCtaSmem|\b%s = [^;]*kOneCtaSmem" % (smem, smem), s), (p, smem)
            seen += 1
    assert seen == 4
