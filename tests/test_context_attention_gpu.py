"""b200_context_attention (csrc/context_attention.cu: tcgen05 S = QK^T into TMEM, fp32 online softmax,
P V with V as an MN-major operand) against the CPU oracle's reference-order sequence
(context_attention.cpp:136-161: RepeatKV -> QK^T -> scale+mask+softmax -> PV -> transpose / remove
padding) on the same seeded inputs, fp16, rel err <= 2e-2; at the cfg3 size
(4 x 2048 tokens, 32 heads) against the unfused GPU sequence of the same library, which the oracle
pins at small sizes (test_parity_gpu.py)."""
import numpy as np
import pytest
import torch

from conftest import assert_close
from oracle import cpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(pkg):
    return pkg.ops


def f16(a):
    return np.ascontiguousarray(np.asarray(a, np.float32).astype(np.float16).astype(np.float32))


def oracle_attention(q, kc, vc, lens, hist):
    """q [B,h,S,d]; kc/vc [1,B,hk,max_seq,d] -> out [Nt, h*d] (fp32 math, P rounded as the reference stores it)"""
    B, h, S, d = q.shape
    lens, hist = np.asarray(lens, np.int32), np.asarray(hist, np.int32)
    ctx = (lens + hist).astype(np.int32)
    Sk, Nt = int(ctx.max()), int(lens.sum())
    pad = np.zeros((B, S), np.int32)
    cum = np.zeros(B + 1, np.int32)
    cpu.cal_padding_offset(pad, cum, lens)
    pad_flat = np.ascontiguousarray(pad.reshape(-1)[:Nt])
    mask = np.zeros((B, S, Sk), np.float32)
    cpu.build_causal_mask(mask, lens, ctx, True)
    kr = np.zeros((B, h, Sk, d), np.float32)
    vr = np.zeros((B, h, Sk, d), np.float32)
    cpu.repeat_kv(kc, kr, 0, ctx)
    cpu.repeat_kv(vc, vr, 0, ctx)
    qk = np.zeros((B, h, S, Sk), np.float32)
    cpu.batched_gemm(q, kr, qk, True)
    cpu.scale_mask_softmax(qk, mask, qk, float(1.0 / np.sqrt(np.float32(d))))
    pv = np.zeros((B, h, S, d), np.float32)
    cpu.batched_gemm(qk, vr, pv, False)
    out = np.zeros((Nt, h * d), np.float32)
    cpu.transpose_remove_padding(pv, out, pad_flat)
    return out, pad_flat


CASES = [
    # h, hk, S (max_q_len), max_seq, lens, hist
    (2, 2, 128, 128, [128], [0]),                 # exactly one tile
    (2, 2, 7, 48, [7], [0]),                      # tiny, ragged
    (4, 2, 16, 64, [5, 16, 9], [0, 0, 0]),        # padding + GQA
    (4, 1, 40, 200, [33, 40], [100, 17]),         # history: first query already sees 100 keys
    (2, 2, 300, 320, [300, 131], [0, 0]),         # three query tiles, diagonal tiles, ragged tails
    (8, 2, 256, 700, [256, 200], [400, 129]),     # history spanning several key tiles
    (2, 1, 1024, 1024, [1024], [0]),              # 8 x 8 tiles
]


@pytest.mark.parametrize("h,hk,S,max_seq,lens,hist", CASES)
def test_context_attention_vs_oracle(ops, h, hk, S, max_seq, lens, hist):
    d, B = 128, len(lens)
    rng = np.random.default_rng(S * 7 + h)
    q = f16(rng.uniform(-1, 1, (B, h, S, d)))
    for b, n in enumerate(lens):
        q[b, :, n:] = 0                              # padded rows are zero-filled by the layer
    kc = f16(rng.uniform(-1, 1, (1, B, hk, max_seq, d)))
    vc = f16(rng.uniform(-1, 1, (1, B, hk, max_seq, d)))
    want, pad_flat = oracle_attention(q, kc, vc, lens, hist)
    # rows at or beyond the context length must not matter, whatever they hold (uninitialised cache)
    kg, vg = kc.copy(), vc.copy()
    for b in range(B):
        kg[0, b, :, lens[b] + hist[b]:] = np.nan
        vg[0, b, :, lens[b] + hist[b]:] = np.inf
    dev = lambda a, dt=torch.float16: torch.from_numpy(np.ascontiguousarray(a)).to("cuda").to(dt)
    out = torch.full((int(sum(lens)), h * d), 7.0, dtype=torch.float16, device="cuda")
    ops.context_attention(dev(q), dev(kg[0]), dev(vg[0]), out, dev(pad_flat, torch.int32),
                          dev(np.asarray(lens, np.int32), torch.int32), dev(np.asarray(hist, np.int32), torch.int32))
    torch.cuda.synchronize()
    assert_close(out.float().cpu().numpy(), want, "fp16", "context attention")


def test_context_attention_rejects_unsupported(ops):
    """fp32 and head sizes other than 128 are not tensor-core shapes: B200_EUNSUPPORTED, no launch"""
    z = lambda *s, dt=torch.float32: torch.zeros(*s, dtype=dt, device="cuda")
    li = torch.tensor([4], dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="unsupported"):
        ops.context_attention(z(1, 2, 4, 128), z(1, 2, 8, 128), z(1, 2, 8, 128), z(4, 256), li, li, li)
    h16 = torch.float16
    with pytest.raises(RuntimeError, match="unsupported"):
        ops.context_attention(z(1, 2, 4, 64, dt=h16), z(1, 2, 8, 64, dt=h16), z(1, 2, 8, 64, dt=h16),
                              z(4, 128, dt=h16), li, li, li)


def test_context_attention_cfg3_vs_unfused_gpu_sequence(ops):
    """cfg3 geometry for one layer (B 4 x S 2048, 32 heads): the flash kernel against the
    library's own reference-order sequence (materialised scores), and the all-ones-V property:
    softmax rows sum to l / (l + 1e-6), so with V = 1 every output element is 1 within fp16 rounding."""
    B, h, hk, S, d = 4, 32, 32, 2048, 128
    g = torch.Generator(device="cuda").manual_seed(5)
    q = (torch.rand(B, h, S, d, device="cuda", generator=g) * 2 - 1).half()
    kc = (torch.rand(B, hk, S, d, device="cuda", generator=g) * 2 - 1).half()
    vc = (torch.rand(B, hk, S, d, device="cuda", generator=g) * 2 - 1).half()
    lens = torch.full((B,), S, dtype=torch.int32, device="cuda")
    hist = torch.zeros(B, dtype=torch.int32, device="cuda")
    pad = torch.zeros(B * S, dtype=torch.int32, device="cuda")
    out = torch.zeros(B * S, h * d, dtype=torch.float16, device="cuda")
    ops.context_attention(q, kc, vc, out, pad, lens, hist)
    # unfused sequence, one sequence at a time to bound the score buffer (h*S*S*2 B = 268 MB)
    mask = torch.zeros(1, S, S, dtype=torch.float16, device="cuda")
    ops.launchBuildCausalMasks(mask, lens[:1], lens[:1])
    for b in range(B):
        qk = torch.empty(1, h, S, S, dtype=torch.float16, device="cuda")
        ops.launchLinearStridedBatchGemm(q[b:b + 1], kc[b:b + 1], qk, False, True)
        ops.launchScaleMaskAndSoftmax(qk, mask, qk, float(1.0 / np.sqrt(d)))
        pv = torch.empty(1, h, S, d, dtype=torch.float16, device="cuda")
        ops.launchLinearStridedBatchGemm(qk, vc[b:b + 1], pv, False, False)
        want = pv[0].permute(1, 0, 2).reshape(S, h * d).float().cpu().numpy()
        assert_close(out[b * S:(b + 1) * S].float().cpu().numpy(), want, "fp16", f"cfg3 sequence {b}")
        del qk, pv
    ones = torch.ones_like(vc)
    ops.context_attention(q, kc, ones, out, pad, lens, hist)
    torch.cuda.synchronize()
    o = out.float()
    assert float((o - 1).abs().max()) <= 2e-3
