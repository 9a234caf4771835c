"""GPU parity tests, model level: the host graph builder (host/gemma_model.cpp) driving the C-ABI layer
versus the CPU oracle's restatement of the reference forward pass (the scalar ggml order), on identical
synthetic weights.  Every comparison is a comparison of BITS."""
import os

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


SMALL = {
    "mqa": dict(n_embd=256, n_layer=3, n_head=4, n_head_kv=1, head_dim=64, n_ff=1024, n_vocab=2048, n_ctx=96),
    # Gemma-7B-like: MHA, n_head*head_dim != n_embd, K > 4096 in the down projection (several K segments: row-lane chain)
    "mha": dict(n_embd=512, n_layer=2, n_head=4, n_head_kv=4, head_dim=128, n_ff=4608, n_vocab=1024, n_ctx=64),
    # K = 3072 as in Gemma-7B: 96 blocks = one full 64-block segment + a short one (quad passes, kf = 1); n_ff = 1280:
    # 40 blocks, a short segment too long for a quad pass (zero-padded plain pass).  The configs above cover kf = 0
    # (K <= 1024) and kf = 2 (n_ff 4608)
    "k96": dict(n_embd=3072, n_layer=1, n_head=2, n_head_kv=2, head_dim=128, n_ff=1280, n_vocab=512, n_ctx=48),
    # every K a multiple of 2048 (64-block segments only), as in Gemma-2B: the plain (non-quad) instantiation of the
    # persistent kernel, which the configs above never reach (their short K rows all take the quad layout)
    "plain": dict(n_embd=2048, n_layer=1, n_head=8, n_head_kv=1, head_dim=256, n_ff=4096, n_vocab=512, n_ctx=48),
    # many rows per CTA in a multi-segment phase (rows > 32: accumulators handed from chain warp to chain warp)
    "wide": dict(n_embd=3072, n_layer=1, n_head=2, n_head_kv=2, head_dim=128, n_ff=1024, n_vocab=16384, n_ctx=48),
    # fewer row pairs than CTAs in a multi-segment phase (DOWN: 128 pairs, K = 4096 = two segments): CTAs WITHOUT rows in
    # the segment-driven row-lane chain - what tensor parallel at 8 ranks does to Gemma-2B (that case once hung)
    "thin": dict(n_embd=256, n_layer=2, n_head=4, n_head_kv=1, head_dim=64, n_ff=4096, n_vocab=1024, n_ctx=48),
    # outside the fused kernel's envelope (n_embd % 256 != 0): exercises the per-operator lowering
    "odd": dict(n_embd=384, n_layer=2, n_head=4, n_head_kv=2, head_dim=96, n_ff=1056, n_vocab=777, n_ctx=48),
}


def _models(gpu, dims, wtype, capture=True, sigma_embd=0.002, fused=True):
    cfg = gpu.make_config(wtype=wtype, sigma_embd=sigma_embd, **dims)
    m = gpu.GemmaModel(cfg)
    m.init_synthetic_weights()
    m.init_kv_cache()
    m.build_compute_graph(capture_acts=capture, fused=fused)
    om = O.Model(wtype=wtype, sigma_embd=sigma_embd, **dims)
    return m, om


@pytest.mark.parametrize("fused", [True, False], ids=["fused", "ops"])
@pytest.mark.parametrize("name", ["mqa", "mha", "k96", "plain", "wide", "thin", "odd"])
@pytest.mark.parametrize("wtype", [O.TYPE_Q4_0, O.TYPE_Q8_0])
def test_generate_matches_oracle(gpu, name, wtype, fused):
    """Prompt (crossing a 32-position chunk boundary) + greedy tokens: ids, every named intermediate of the last
    step, the logits and the KV cache are BIT-IDENTICAL to the oracle (scalar ggml order), through the persistent
    kernel and through the per-operator kernels."""
    dims = SMALL[name]
    m, om = _models(gpu, dims, wtype, fused=fused)
    assert m.is_fused == (fused and name != "odd")
    if m.is_fused:  # the computed soft-max exp must have been proved identical to the fp16 table on this GPU
        assert m.exp_computed
    prompt = ((1 + 7919 * np.arange(35)) % dims["n_vocab"]).astype(np.int32)
    n_decode = 8
    toks, _, _ = m.generate(prompt, n_decode)
    rtoks, _, _ = om.generate(prompt, n_decode, O.REF)
    assert np.array_equal(toks, rtoks)
    for il in range(dims["n_layer"]):
        for cap in ("kqv_out", "sa_out", "ffn_act", "l_out"):
            assert np.array_equal(bits(m.capture(cap, il)), bits(om.capture(cap, il))), (cap, il)
    assert np.array_equal(bits(m.capture("result_norm")), bits(om.capture("result_norm")))
    assert np.array_equal(bits(m.logits()), bits(om.capture("result_output")))
    for il in range(dims["n_layer"]):
        gk, gv = m.kv(il)
        ok, ov = om.kv(il)
        n = len(prompt) + n_decode - 1
        assert np.array_equal(gk[:n], ok[:n]) and np.array_equal(gv[:n], ov[:n])
    m.close()
    om.close()


@pytest.mark.parametrize("wname", ["q8_0", "q4_0"])
def test_config1_full_size_greedy_stream(gpu, wname):
    """A greedy stream at FULL size: Gemma-2B, 128-token prompt id_i = (1 + 7919 i) mod V, 64 greedy tokens,
    against the oracle's run of the reference CPU path (tests/golden/config1_2b_*.npz, made by
    tests/golden/make_config1.py; loop of ref: src/gemma_model.cpp:548-575).  The stream is NOT degenerate
    (sigma_embd = 0.004: 64 distinct ids, top-2 margins down to 4e-5 of |logit| ~ 0.85), so it is reproduced only by
    arithmetic that matches the reference's bit for bit: all 64 ids, and the 16 largest + 1024 sampled logits of
    every step must be identical."""
    z = np.load(os.path.join(GOLDEN, f"config1_2b_{wname}.npz"))
    wtype = O.TYPE_Q8_0 if wname == "q8_0" else O.TYPE_Q4_0
    dims = dict(gpu.GEMMA_2B, n_ctx=int(z["n_ctx"]))
    m = gpu.GemmaModel(gpu.make_config(wtype=wtype, sigma_embd=float(z["sigma_embd"]), **dims))
    m.init_synthetic_weights()
    m.init_kv_cache()
    m.build_compute_graph(capture_acts=False)
    assert m.is_fused
    prompt = z["prompt"]
    assert len(set(z["tokens"].tolist())) >= 32  # the fixture itself: a non-degenerate stream
    margins = z["top_val"][:, 0] - z["top_val"][:, 1]
    for t, tok in enumerate(prompt[:-1]):
        m.decode_step(int(tok), t)
    tok, pos = int(prompt[-1]), len(prompt) - 1
    for s in range(len(z["tokens"])):
        tok = m.decode_step(tok, pos)
        pos += 1
        lg = m.logits()
        assert tok == int(z["tokens"][s]), f"step {s}: token {tok} != {int(z['tokens'][s])} (top-2 margin {margins[s]:.2e})"
        assert np.array_equal(bits(lg[z["top_idx"][s]]), bits(z["top_val"][s])), f"step {s}: top-16 logits differ"
        assert np.array_equal(bits(lg[z["sample_idx"]]), bits(z["sample_val"][s])), f"step {s}: sampled logits differ"
    out_dir = os.path.join(os.path.dirname(GOLDEN), "..", "build", "reports")
    if os.path.isdir(out_dir):
        import json
        json.dump(dict(config="gemma-2b %s, 128-token prompt + 64 greedy tokens" % wname, tokens_identical=64,
                       logits="bit-identical (top-16 + 1024 sampled per step)", min_top2_margin=float(margins.min()),
                       median_top2_margin=float(np.median(margins)), mean_absmax_logit=float(z["absmax"].mean()),
                       max_abs_deviation=0.0, distinct_tokens=len(set(z["tokens"].tolist()))),
                  open(os.path.join(out_dir, f"config1_parity_{wname}.json"), "w"))
    m.close()


def test_uploaded_weights_equal_synthetic_weights(gpu):
    """set_tensor(host AoS blocks from the oracle) gives the same model as on-device generation."""
    dims = SMALL["mqa"]
    m, om = _models(gpu, dims, O.TYPE_Q4_0)
    prompt = np.array([5, 9, 200, 31], dtype=np.int32)
    t1, _, _ = m.generate(prompt, 4)
    l1 = m.logits()
    n_tensors = 2 + 9 * dims["n_layer"]
    for tid in range(n_tensors):
        raw, rows, cols = om.tensor(tid)
        m.set_tensor(tid, raw)
    m.build_compute_graph(capture_acts=True)
    t2, _, _ = m.generate(prompt, 4)
    assert np.array_equal(t1, t2) and np.array_equal(bits(l1), bits(m.logits()))
    m.close()
    om.close()


def test_device_resident_loop_equals_host_stepped_loop(gpu):
    """run_steps (no host round trip, token fed back on the device) == decode_step per token; stepping past the
    context is refused on the host and the device position stops at n_ctx - 1."""
    dims = SMALL["mqa"]
    m, om = _models(gpu, dims, O.TYPE_Q8_0, capture=False)
    prompt = np.array([7, 8, 9], dtype=np.int32)
    toks, _, _ = m.generate(prompt, 9)
    m.init_kv_cache()
    for t, tok in enumerate(prompt[:-1]):
        m.decode_step(tok, t)
    m.set_state(int(prompt[-1]), len(prompt) - 1, 1)
    m.run_steps(9)
    gpu.sync()
    tok, pos = m.get_state()
    assert tok == toks[-1] and pos == len(prompt) - 1 + 9
    m.set_state(5, dims["n_ctx"] - 2, 1)
    m.run_steps(2)  # positions n_ctx - 2 and n_ctx - 1: allowed
    gpu.sync()
    assert m.get_state()[1] == dims["n_ctx"] - 1  # the device position saturates
    with pytest.raises(gpu.GgbError):
        m.set_state(5, dims["n_ctx"] - 2, 1)
        m.run_steps(3)
    m.close()
    om.close()


def test_pinned_position_is_idempotent(gpu):
    """pos_step = 0 (fixed n_kv, used by bench.py): repeating a step reproduces the same logits."""
    dims = SMALL["mqa"]
    m, om = _models(gpu, dims, O.TYPE_Q4_0, capture=False)
    m.fill_kv_cache_synthetic(3)
    m.set_state(11, dims["n_ctx"] - 1, 0)
    m.run_steps(1)
    gpu.sync()
    l1, t1 = m.logits(), m.get_state()
    m.set_state(11, dims["n_ctx"] - 1, 0)
    m.run_steps(1)
    gpu.sync()
    assert np.array_equal(bits(l1), bits(m.logits())) and t1 == m.get_state()
    m.close()
    om.close()


# ---------------------------------------------------------------- full-size checks without a full-size oracle run
def _q8(x):
    return O.quantize(O.TYPE_Q8_0, np.ascontiguousarray(x, dtype=np.float32)[None, :])


def _rows(seed, tid, rows, k, wtype, sigma=0.02):
    """the oracle's generator + quantiser for sampled rows of a synthetic weight matrix"""
    return np.stack([O.quantize(wtype, O.synth_row(seed, tid, int(r), k, sigma)[None, :])[0] for r in rows])


def _full_size_checks(gpu, dims, wtype, pos, token=4242):
    """One decode step at full size with a synthetic KV cache, re-derived piece by piece on the oracle from the GPU's own
    intermediates (so no full-size oracle forward is needed), everything compared bit for bit:
      embedding row -> attn_norm -> Q8_0 -> Wq / Wk / Wv rows of one head -> rope -> kq over ALL positions ->
      soft_max_ext -> fp16 P . V  == kqv_out[0] of that head            (SCORE + PV phases at the real context length)
      sa_out[0]   == Wo . Q8_0(kqv_out[0]) + x0 on sampled rows          (O phase)
      ffn_act[0]  == gelu(Wg . a) * (Wu . a), a = Q8_0(ffn_norm(sa_out[0])), on sampled rows   (GATE_UP + GeGLU)
      l_out[0]    == Wd . Q8_0(ffn_act[0]) + sa_out[0] on sampled rows   (DOWN: the longest K)
      logits      == E . Q8_0(result_norm) on sampled rows, token == first maximum (LOGITS + SAMPLE)"""
    cfg = gpu.make_config(wtype=wtype, **dims)
    m = gpu.GemmaModel(cfg)
    m.init_synthetic_weights()
    m.init_kv_cache()
    m.fill_kv_cache_synthetic(99)
    m.build_compute_graph(capture_acts=True)
    assert m.is_fused
    E, H, Hkv, d, F, V = (dims[k] for k in ("n_embd", "n_head", "n_head_kv", "head_dim", "n_ff", "n_vocab"))
    seed, eps = cfg.seed, cfg.eps
    m.set_state(token, pos, 0)
    m.run_steps(1)
    gpu.sync()
    logits = m.logits()
    tok, p = m.get_state()
    assert p == pos and tok == O.argmax(logits)
    m.set_state(token, pos, 0)
    m.run_steps(1)
    gpu.sync()
    assert np.array_equal(bits(logits), bits(m.logits()))  # deterministic at a pinned position

    T = O.tensor_id
    norm_w = lambda tid: O.synth_row(seed, tid, 0, E, 0.02, 1.0)
    # x0 = get_rows(token_embd, token) * sqrt(E)
    x0 = O.dequantize(wtype, _rows(seed, 0, [token], E, wtype), E)[0] * np.float32(np.sqrt(np.float32(E)))
    a0 = _q8(O.rms_norm(x0, eps) * norm_w(T(0, 0)))
    # ---- attention of one head over the whole context
    h = H - 1
    g = h // (H // Hkv)
    hr = np.arange(h * d, (h + 1) * d)
    gr = np.arange(g * d, (g + 1) * d)
    q = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 1), hr, E, wtype), a0, E)[0]
    k = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 2), gr, E, wtype), a0, E)[0]
    v = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 3), gr, E, wtype), a0, E)[0]
    q_r = O.rope_neox(q[None, :], pos) * np.float32(1.0 / np.sqrt(np.float32(d)))
    gk, gv = m.kv(0)
    kv_heads = gk.shape[1] // d
    kc = np.ascontiguousarray(gk[:, g * d:(g + 1) * d] if kv_heads == Hkv else gk[:, :d])
    vc = np.ascontiguousarray(gv[:, g * d:(g + 1) * d] if kv_heads == Hkv else gv[:, :d])
    # the new position's rows were written by the kernel: compare them, then use the cache as it is
    assert np.array_equal(kc[pos], O.rope_neox(k[None, :], pos).astype(np.float16).view(np.uint16)[0])
    assert np.array_equal(vc[pos], v.astype(np.float16).view(np.uint16))
    want = O.attn_decode(O.REF, q_r, kc, vc, pos + 1, dims["n_ctx"])[0]
    kqv = m.capture("kqv_out", 0)
    assert np.array_equal(bits(kqv[hr]), bits(want)), f"attention head {h}: max abs {np.abs(kqv[hr] - want).max()}"
    # ---- O, GATE_UP (+ GeGLU), DOWN, LOGITS on sampled rows
    sa = m.capture("sa_out", 0)
    rows = np.r_[0:8, E // 2:E // 2 + 8, E - 8:E]
    want = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 4), rows, H * d, wtype), _q8(kqv), H * d)[0] + x0[rows]
    assert np.array_equal(bits(sa[rows]), bits(want))
    af = _q8(O.rms_norm(sa, eps) * norm_w(T(0, 5)))
    act = m.capture("ffn_act", 0)
    frows = np.r_[0:8, F // 2 + 5:F // 2 + 13, F - 8:F]
    gate = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 6), frows, E, wtype), af, E)[0]
    up = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 7), frows, E, wtype), af, E)[0]
    assert np.array_equal(bits(act[frows]), bits(O.gelu(gate) * up))
    lo = m.capture("l_out", 0)
    want = O.mul_mat(wtype, O.REF, _rows(seed, T(0, 8), rows, F, wtype), _q8(act), F)[0] + sa[rows]
    assert np.array_equal(bits(lo[rows]), bits(want))
    vrows = np.r_[0:32, V // 2:V // 2 + 32, V - 32:V]
    want = O.mul_mat(wtype, O.REF, _rows(seed, 0, vrows, E, wtype), _q8(m.capture("result_norm")), E)[0]
    assert np.array_equal(bits(logits[vrows]), bits(want))
    wb = m.weight_bytes
    m.close()
    return wb


def test_full_size_gemma_2b_q4_0(gpu):
    """BASELINE config 2 at full size (Gemma-2B, Q4_0, n_kv = 2048)."""
    wb = _full_size_checks(gpu, dict(gpu.GEMMA_2B, n_ctx=2048), O.TYPE_Q4_0, 2047)
    assert wb == 1409679360  # algorithmic bytes for 2B Q4_0


def test_full_size_gemma_7b_q4_0(gpu):
    """BASELINE config 4 shape at full size (Gemma-7B, Q4_0, n_kv = 2048): quad passes (K = 3072), MHA, 16 KV heads."""
    wb = _full_size_checks(gpu, dict(gpu.GEMMA_7B, n_ctx=2048), O.TYPE_Q4_0, 2047)
    assert wb == 4802347008


def test_full_size_gemma_7b_q8_0_ctx8192(gpu):
    """BASELINE config 5 at its longest context (Gemma-7B, Q8_0, n_kv = 8192)."""
    wb = _full_size_checks(gpu, dict(gpu.GEMMA_7B, n_ctx=8192), O.TYPE_Q8_0, 8191)
    assert wb == 9071099904
