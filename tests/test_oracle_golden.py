"""Pins the CPU oracle (oracle/llama_cpu.c) to the reference:
 * against tests/golden/ref_cpu_golden.npz — outputs of the reference's own unit-test CPU
   functions on the reference tests' own data (generated by tests/golden/make_golden.py), and the
   golden vector written in tests/unittests/test_cal_paddingoffset.cu:54-56;
 * against closed forms the reference tests imply.
Runs on CPU (no `gpu` marker)."""
import os

import numpy as np
import pytest

from oracle import cpu

G = np.load(os.path.join(os.path.dirname(__file__), "golden", "ref_cpu_golden.npz"))


def test_rmsnorm_reference_vector():
    # tests/unittests/test_rmsnorm.cu:139-192
    nt, H = 64, 4096
    x = (np.arange(nt * H) % 2 + 1).astype(np.float32).reshape(nt, H)
    g = (np.arange(H) % 2 + 1).astype(np.float32)
    res = np.zeros_like(x)
    x0 = x.copy()
    cpu.rmsnorm(x, res, g, 1e-6)
    assert np.max(np.abs(x[0] - G["rmsnorm_row0"])) <= 1e-6   # the reference's own 1e-6 check (:58)
    assert np.max(np.abs(x[63] - G["rmsnorm_row63"])) <= 1e-6
    assert np.array_equal(res, x0)                            # residual = pre-norm input (D7)
    # closed form: mean(x^2) = 2.5 -> x*gamma/sqrt(2.5+eps)
    want = x0[0] * g / np.sqrt(2.5 + 1e-6)
    assert np.allclose(x[0], want, rtol=1e-6)


def test_fused_add_norm_reference_vector():
    # tests/unittests/test_fused_addresidual_norm.cu:69-141  -> every output is 1/sqrt(1.5)
    o = np.ones((2, 32), np.float32)
    r = np.zeros((2, 32), np.float32)
    cpu.fused_add_bias_residual_rmsnorm(r, o, np.zeros(32, np.float32), np.ones(32, np.float32), 0.5)
    assert np.max(np.abs(o - G["addnorm_out"])) <= 1e-6
    assert np.allclose(o, 1 / np.sqrt(1.5), rtol=1e-6)
    assert np.array_equal(r, np.ones((2, 32), np.float32))


def test_swiglu_reference_vectors():
    # tests/unittests/test_act.cu:46-57
    gi = np.ones((16, 2, 11008), np.float32)
    go = np.zeros((16, 11008), np.float32)
    cpu.swiglu(gi, go)
    assert np.max(np.abs(go.reshape(-1)[:8] - G["swiglu_first8"])) <= 1e-6
    assert np.allclose(go, 1 / (1 + np.exp(-1.0)), rtol=1e-6)
    gi = G["swiglu_ramp_in"].copy()
    go = np.zeros((2, 64), np.float32)
    cpu.swiglu(gi, go)
    assert np.max(np.abs(go - G["swiglu_ramp_out"])) <= 1e-6


def test_rope_prefill_reference_vector():
    # tests/unittests/test_bias_and_RoPE.cu:99-160 (constant 32.0 data; CPUfunc is token-major
    # [B,S,h,d], ours is the kernel's [B,h,S,d]; with constant data every head is identical)
    B, S, h, hk, d = 1, 32, 32, 32, 128
    q = np.zeros((B, h, S, d), np.float32)
    k = np.zeros((B, hk, S, d), np.float32)
    v = np.zeros((B, hk, S, d), np.float32)
    QKV = np.full((B * S, h + 2 * hk, d), 32.0, np.float32)
    cpu.qkv_bias_rope_transpose(q, k, v, QKV, None, np.zeros(B * S, np.int32),
                                np.zeros(B, np.int32), 128, 10000.0)
    for head in (0, 17, 31):
        assert np.max(np.abs(q[0, head] - G["rope_q_head0"])) <= 2e-5 * 32
        assert np.max(np.abs(k[0, head] - G["rope_k_head0"])) <= 2e-5 * 32
    assert np.array_equal(v, np.full_like(v, 32.0))


def test_rope_decode_matches_prefill_row():
    # decode RoPE at step s+1 == prefill row s (same formula, qkv_bias_and_RoPE.cu:29-46)
    rng = np.random.default_rng(0)
    h, hk, d = 4, 2, 16
    tok = rng.standard_normal((1, h + 2 * hk, d)).astype(np.float32)
    S = 6
    QKV = np.repeat(tok, S, axis=0)
    q = np.zeros((1, h, S, d), np.float32)
    k = np.zeros((1, hk, S, d), np.float32)
    v = np.zeros((1, hk, S, d), np.float32)
    cpu.qkv_bias_rope_transpose(q, k, v, QKV, None, np.zeros(S, np.int32), np.zeros(1, np.int32),
                                d, 10000.0)
    for s in range(S):
        t = tok.copy()
        cpu.rope_decode(t, h, hk, s + 1, d, 10000.0)
        assert np.array_equal(t[0, :h], q[0, :, s])
        assert np.array_equal(t[0, h:h + hk], k[0, :, s])
        assert np.array_equal(t[0, h + hk:], tok[0, h + hk:])


def test_linear_reference_vector():
    # tests/unittests/test_linear.cu:39-60 (integer data: exact in fp32)
    m, kk, n = 13, 4096, 64
    a = (np.arange(m * kk) % 3).astype(np.float32).reshape(m, kk)
    w_full_cols = (np.arange(kk * 4096) % 3).astype(np.float32).reshape(kk, 4096)[:, :n].copy()
    y = np.zeros((m, n), np.float32)
    cpu.linear(a, w_full_cols, y, trans_b=False)
    assert np.array_equal(y, G["linear_cols64"])
    y2 = np.zeros((m, n), np.float32)
    cpu.linear(a, np.ascontiguousarray(w_full_cols.T), y2, trans_b=True)
    assert np.array_equal(y2, y)


def test_causal_mask_reference_vectors():
    mask = np.zeros((1, 5, 5), np.float32)
    cpu.build_causal_mask(mask, np.array([5], np.int32), np.array([5], np.int32), True)
    assert np.array_equal(mask, G["mask_5x5"])
    assert np.array_equal(mask[0], np.tril(np.ones((5, 5), np.float32)))
    # the GPU kernel's extra clause agrees when klen == qlen
    m2 = np.zeros((1, 5, 5), np.float32)
    cpu.build_causal_mask(m2, np.array([5], np.int32), np.array([5], np.int32), False)
    assert np.array_equal(m2, mask)
    mask = np.zeros((2, 4, 7), np.float32)
    cpu.build_causal_mask(mask, np.array([3, 4], np.int32), np.array([6, 4], np.int32), True)
    assert np.array_equal(mask, G["mask_hist"])


def test_padding_offset_golden_vector():
    # tests/unittests/test_cal_paddingoffset.cu:13-14,32,54-56
    pad = np.full((3, 5), -1, np.int32)
    cum = np.zeros(4, np.int32)
    cpu.cal_padding_offset(pad, cum, np.array([3, 3, 3], np.int32))
    assert np.array_equal(pad.reshape(-1)[:9], G["padding_offset_golden"])
    assert np.array_equal(cum, G["cum_seqlens_golden"])
    assert np.all(pad.reshape(-1)[9:] == -1)   # entries past the token count are not written


def test_copies_ragged_and_empty():
    rng = np.random.default_rng(1)
    layers, B, hk, h, S, max_seq, d = 2, 3, 2, 4, 5, 9, 8
    src = rng.standard_normal((B, hk, S, d)).astype(np.float16)
    cache = np.zeros((layers, B, hk, max_seq, d), np.float16)
    cur = np.array([5, 0, 2], np.int32)      # includes an empty sequence
    hist = np.array([1, 3, 4], np.int32)
    cpu.concat_kv(src, cache, 1, cur, hist)
    assert not cache[0].any()
    for b in range(B):
        assert np.array_equal(cache[1, b, :, hist[b]:hist[b] + cur[b]], src[b, :, :cur[b]])
        assert not cache[1, b, :, :hist[b]].any() and not cache[1, b, :, hist[b] + cur[b]:].any()
    ctx = (cur + hist).astype(np.int32)
    dst = np.full((B, h, 8, d), 7, np.float16)
    cpu.repeat_kv(cache, dst, 1, ctx)
    for b in range(B):
        for j in range(h):
            assert np.array_equal(dst[b, j, :ctx[b]], cache[1, b, j // 2, :ctx[b]])
            assert np.all(dst[b, j, ctx[b]:] == 7)


def test_softmax_matches_numpy():
    # tests/unittests/test_mask_softmax.cu:60-65 shapes: B=1, h=2, 8x8, data i%8, mask=1
    qk = (np.arange(2 * 64) % 8).astype(np.float32).reshape(1, 2, 8, 8)
    mask = np.ones((1, 8, 8), np.float32)
    out = np.zeros_like(qk)
    cpu.scale_mask_softmax(qk, mask, out, 0.5)
    s = 0.5 * qk
    e = np.exp(s - s.max(-1, keepdims=True))
    assert np.allclose(out, e / (e.sum(-1, keepdims=True) + 1e-6), rtol=1e-6)


def test_decode_attention_vs_numpy_gqa():
    rng = np.random.default_rng(2)
    B, h, hk, d, max_seq, step = 2, 8, 2, 16, 12, 7
    qkv = rng.standard_normal((B, h + 2 * hk, d)).astype(np.float32)
    kc = rng.standard_normal((B, hk, max_seq, d)).astype(np.float32)
    vc = rng.standard_normal((B, hk, max_seq, d)).astype(np.float32)
    out = np.zeros((B, h * d), np.float32)
    cpu.decode_attention(qkv, kc, vc, out, h, hk, step, True)
    assert np.array_equal(kc[:, :, step - 1], qkv[:, h:h + hk])        # appended rows
    assert np.array_equal(vc[:, :, step - 1], qkv[:, h + hk:])
    for b in range(B):
        for j in range(h):
            K, V = kc[b, j // 4, :step], vc[b, j // 4, :step]
            s = (K @ qkv[b, j]) / np.sqrt(d)
            e = np.exp(s - s.max())
            want = (e / (e.sum() + 1e-6)) @ V
            assert np.allclose(out[b, j * d:(j + 1) * d], want, rtol=1e-5, atol=1e-6)


def test_topk_ties_lower_index_first():
    logits = np.array([[1, 5, 5, 3, 5, 0]], np.float32)
    ids = np.zeros((1, 4), np.int32)
    vals = np.zeros((1, 4), np.float32)
    cpu.topk(logits, ids, vals, 4)
    assert ids.tolist() == [[1, 2, 4, 3]]
    assert vals.tolist() == [[5, 5, 5, 3]]


@pytest.mark.skipif(not os.path.exists(os.path.join(os.path.dirname(__file__), "..", "oracle", "_ref", "libref.so")),
                    reason="oracle/_ref not built (needs /root/reference)")
def test_oracle_vs_live_reference_cpu_functions_random():
    """Beyond the fixed vectors: random data through the reference's CPU functions, live."""
    import ctypes as C
    try:
        ref = C.CDLL(os.path.join(os.path.dirname(__file__), "..", "oracle", "_ref", "libref.so"))
    except OSError as e:  # CUDA runtime libs not loadable on this host
        pytest.skip(str(e))
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    rng = np.random.default_rng(3)
    x = rng.standard_normal((7, 512)).astype(np.float32)
    g = rng.standard_normal(512).astype(np.float32)
    a, b = x.copy(), x.copy()
    cpu.rmsnorm(a, None, g, 1e-5)
    ref.ref_cpu_rmsnorm(p(b), p(g), C.c_float(1e-5), 512, 7)
    assert np.max(np.abs(a - b)) / np.max(np.abs(b)) < 1e-6
    gi = rng.standard_normal((3, 2, 96)).astype(np.float32)
    o1, o2 = np.zeros((3, 96), np.float32), np.zeros((3, 96), np.float32)
    cpu.swiglu(gi, o1)
    ref.ref_cpu_swiglu(p(gi), p(o2), 3, 96)
    assert np.max(np.abs(o1 - o2)) < 1e-6
    xm = rng.standard_normal((5, 64)).astype(np.float32)
    w = rng.standard_normal((64, 48)).astype(np.float32)
    y1, y2 = np.zeros((5, 48), np.float32), np.zeros((5, 48), np.float32)
    cpu.linear(xm, w, y1, trans_b=False)
    ref.ref_cpu_linear(p(xm), p(w), p(y2), 5, 64, 48)
    assert np.max(np.abs(y1 - y2)) / np.max(np.abs(y2)) < 1e-5
