"""Latent attention of prompt portions on tcgen05 tiles: portions that end at, before and behind a tile of rows, contexts around a tile of keys."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("heads,W,cols,PR,window,sink,sign", [(16, 576, 512, 64, 0, False, 1.0), (5, 640, 512, 128, 0, True, 1.0), (20, 320, 256, 64, 100, True, 1.0),
                                                              (64, 512, 512, 64, 33, False, -1.0), (1, 256, 256, 64, 0, False, 1.0), (16, 576, 512, 64, 0, True, 1.0)])
@pytest.mark.parametrize("several", [True, False])
@pytest.mark.parametrize("round_q", [False, True])
def test_prompt_portions_on_tiles(S, heads, W, cols, PR, window, sink, sign, several, round_q):
    """the query is a bfloat16 operand: independent errors of 2^-9 in every score term, about 2e-3 of the result's norm; 8e-3 is four times
    that. A query of bfloat16 numbers leaves the weights (the sum of two bfloat16, off by 2^-18 of a weight on average) and the sums (2 * 700 / 16 additions of
    the tensor core, each off by at most 2^-23): 3e-5. Rows nobody owns are NaN: reading one into a sum would show"""
    g = torch.Generator().manual_seed(W + heads)
    TQ = 128 // heads
    # (rows in the cache before the portion, rows of the portion)
    entries = [(0, 1), (63, 2), (5, TQ - 1), (0, TQ), (64, TQ + 1), (700, 1), (1, 65)] if several else [(61, 2 * TQ + 3)]
    entries = [(p, n) for p, n in entries if n > 0]
    lens = [p + n for p, n in entries]
    need = [(n + PR - 1) // PR for n in lens]
    order = torch.randperm(sum(need) + 1, generator=g).tolist()
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    pool = torch.full(((sum(need) + 1) * PR, W), float("nan"))
    rows = [torch.randn(n, W, generator=g).bfloat16().double() for n in lens]
    for b, n in enumerate(lens):
        for i in range(need[b]):
            pg, m = order.pop(), min(PR, n - i * PR)
            table[b, i] = pg
            pool[pg * PR:pg * PR + m] = rows[b][i * PR:i * PR + m]
    slot = torch.cat([torch.full((n,), b, dtype=torch.int32) for b, (p, n) in enumerate(entries)])
    pos = torch.cat([torch.arange(p, p + n, dtype=torch.int32) for p, n in entries])
    T, scale = slot.numel(), sign * 0.9 * W ** -0.5
    qa, sk = torch.randn(T, heads, W, generator=g), torch.randn(heads, generator=g) * 2
    qa = qa.bfloat16().float() if round_q else qa
    dev = [x.cuda().contiguous() for x in (qa, pool.bfloat16(), table, slot, pos, sk)]
    out = torch.full((T, heads, W), 7.0, device="cuda")
    a = S.LatentAttentionArgs()
    a.qa, a.out, a.pool, a.pages, a.max_pages, a.page_rows = dev[0].data_ptr(), out.data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), table.shape[1], PR
    a.slot, a.pos, a.sink, a.scale = dev[3].data_ptr(), dev[4].data_ptr(), dev[5].data_ptr() if sink else None, scale
    a.n_tokens, a.heads, a.rank, a.window, a.dtype, a.out_cols = T, heads, W, window, S.BF16, cols
    a.longest_entry, a.longest_context = max(n for p, n in entries), max(lens)
    torch.cuda.synchronize()
    assert S.lib().b200_latent_attention_ex(C.byref(a), None) == 0
    torch.cuda.synchronize()
    got = out.double().cpu()
    if cols < W:
        assert bool((got[:, :, cols:] == 7.0).all())          # columns nobody asked for
    for t in range(T):
        b, p = int(slot[t]), int(pos[t])
        kv = rows[b][max(0, p + 1 - window) if window else 0:p + 1]
        s = qa[t].double() @ kv.T * scale
        top = torch.maximum(s.amax(1, keepdim=True), sk.double()[:, None]) if sink else s.amax(1, keepdim=True)
        e = torch.exp(s - top)
        w = e / (e.sum(1, keepdim=True) + (torch.exp(sk.double()[:, None] - top) if sink else 0.0))
        want = w @ kv[:, :cols]
        assert float((got[t, :, :cols] - want).norm() / want.norm()) < (3e-5 if round_q else 8e-3), (t, b, p)


@pytest.mark.parametrize("heads,W,cols,window", [(16, 576, 512, 0), (8, 320, 256, 0), (8, 320, 256, 600), (64, 512, 512, 0)])
@pytest.mark.parametrize("entries", [[(3990, 2)], [(1500, 16)], [(2100 - 40 * i, 1) for i in range(12)] + [(1990, 16)], [(1400, 4), (1300, 3), (900, 1), (1200, 2)]])
def test_few_rows_behind_long_contexts(pkg, S, heads, W, cols, window, entries):
    """with a workspace and the hints that a model gives: one portion of a few tokens is shared out over the context, single tokens beside a portion
    have a CTA each. A query of bfloat16 numbers; the mma.sync tiles round their weights to bfloat16 (1.2e-3 on average, 5e-3 is four times that)"""
    g = torch.Generator().manual_seed(W + len(entries))
    PR, lens = 64, [p + n for p, n in entries]
    need = [(n + PR - 1) // PR for n in lens]
    order = torch.randperm(sum(need), generator=g)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    rows = [torch.randn(n, W, generator=g).bfloat16().double() for n in lens]
    pool, at = torch.full((sum(need) * PR, W), float("nan")), 0
    for b, n in enumerate(lens):
        table[b, :need[b]] = order[at:at + need[b]].int()
        at += need[b]
        for i in range(need[b]):
            m = min(PR, n - i * PR)
            pool[int(table[b, i]) * PR:int(table[b, i]) * PR + m] = rows[b][i * PR:i * PR + m]
    slot = torch.cat([torch.full((n,), b, dtype=torch.int32) for b, (p, n) in enumerate(entries)])
    pos = torch.cat([torch.arange(p, p + n, dtype=torch.int32) for p, n in entries])
    T, scale, longest = slot.numel(), 0.9 * W ** -0.5, max(n for p, n in entries)
    qa = torch.randn(T, heads, W, generator=g).bfloat16().float()
    dev = [x.cuda().contiguous() for x in (qa, pool.bfloat16(), table, slot, pos)]
    out, ws_bytes = torch.full((T, heads, W), 7.0, device="cuda"), S.lib().b200_latent_attention_workspace_bytes(T, heads, W)
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    a = S.LatentAttentionArgs()
    a.qa, a.out, a.pool, a.pages, a.max_pages, a.page_rows = dev[0].data_ptr(), out.data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), table.shape[1], PR
    a.slot, a.pos, a.scale, a.workspace, a.workspace_bytes = dev[3].data_ptr(), dev[4].data_ptr(), scale, ws.data_ptr(), ws_bytes
    a.n_tokens, a.heads, a.rank, a.window, a.dtype, a.out_cols, a.longest_entry, a.longest_context = T, heads, W, window, S.BF16, cols, longest, max(lens)
    torch.cuda.synchronize()
    before = pkg.capi.lib().b200_launch_count()
    assert S.lib().b200_latent_attention_ex(C.byref(a), None) == 0
    launches = pkg.capi.lib().b200_launch_count() - before
    torch.cuda.synchronize()
    if entries == [(3990, 2)] and not window:
        assert launches == 2          # the shares of the context and their merge
    got = out.double().cpu()
    for t in range(T):
        b, p = int(slot[t]), int(pos[t])
        kv = rows[b][max(0, p + 1 - window) if window else 0:p + 1]
        w = torch.softmax(qa[t].double() @ kv.T * scale, 1)
        want = w @ kv[:, :cols]
        assert float((got[t, :, :cols] - want).norm() / want.norm()) < 5e-3, (t, b, p)
