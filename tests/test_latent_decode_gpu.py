"""Latent attention of single tokens (a cluster per token): contexts that end at, before and behind a half tile, a share and a page."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("heads,W,cols,PR,window,sink", [(16, 576, 512, 64, 0, False), (5, 72, 64, 64, 0, True), (20, 320, 256, 48, 100, True),
                                                         (16, 640, 640, 32, 33, False), (1, 16, 16, 16, 0, False)])
def test_single_tokens_share_their_rows_in_a_cluster(S, heads, W, cols, PR, window, sink):
    """query and weights are bfloat16 operands: independent errors of 2^-9 in every weight and score term, about 2e-3 of the result's
    norm; 8e-3 is four times that. Rows nobody owns are NaN: reading one would show"""
    g = torch.Generator().manual_seed(W + heads)
    lens = [1, 31, 32, 33, 64, 65, 513, 1400]
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
    T, scale = len(lens), 0.9 * W ** -0.5
    qa, sk = torch.randn(T, heads, W, generator=g), torch.randn(heads, generator=g) * 2
    dev = [x.cuda().contiguous() for x in (qa, pool.bfloat16(), table, torch.arange(T, dtype=torch.int32), torch.tensor([n - 1 for n in lens], dtype=torch.int32), sk)]
    for longest in (max(lens), 0):
        out = torch.full((T, heads, W), 7.0, device="cuda")
        a = S.LatentAttentionArgs()
        a.qa, a.out, a.pool, a.pages, a.max_pages, a.page_rows = dev[0].data_ptr(), out.data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), table.shape[1], PR
        a.slot, a.pos, a.sink, a.scale = dev[3].data_ptr(), dev[4].data_ptr(), dev[5].data_ptr() if sink else None, scale
        a.n_tokens, a.heads, a.rank, a.window, a.dtype, a.longest_entry, a.longest_context, a.out_cols = T, heads, W, window, S.BF16, 1, longest, cols
        torch.cuda.synchronize()
        assert S.lib().b200_latent_attention_ex(C.byref(a), None) == 0
        torch.cuda.synchronize()
        got = out.double().cpu()
        assert bool((got[:, :, cols:] == 7.0).all())          # columns nobody asked for
        for b, n in enumerate(lens):
            kv = rows[b][max(0, n - window) if window else 0:]
            s = qa[b].double() @ kv.T * scale
            top = torch.maximum(s.amax(1, keepdim=True), sk.double()[:, None]) if sink else s.amax(1, keepdim=True)
            e = torch.exp(s - top)
            w = e / (e.sum(1, keepdim=True) + (torch.exp(sk.double()[:, None] - top) if sink else 0.0))
            want = w @ kv[:, :cols]
            assert float((got[b, :, :cols] - want).norm() / want.norm()) < 8e-3, (b, n)


@pytest.mark.parametrize("T", [1, 20, 80, 160])
@pytest.mark.parametrize("PR", [64, 48])
def test_weights_of_single_tokens_are_the_sum_of_two_bfloat16(S, T, PR):
    """queries that bfloat16 holds, so what is left is a weight's rounding, 2^-18 of it, and the scores' fp32 sums, 2^-24 * 36 steps of a few units: 1e-5 together, the bound is three
    times that. A weight rounded to one bfloat16 is off by up to 2^-9. Sixteen shares of a context to one"""
    g = torch.Generator().manual_seed(T + PR)
    heads, W, cols, n = 16, 576, 512, 1400
    rows = torch.randn(n, W, generator=g).bfloat16()
    pool = torch.full(((n + PR - 1) // PR * PR, W), float("nan"), dtype=torch.bfloat16)
    pool[:n] = rows
    qa, scale = torch.randn(T, heads, W, generator=g).bfloat16().float(), W ** -0.5
    pos = [n - 1 - i for i in range(T)]
    dev = [qa.cuda(), pool.cuda(), torch.arange(pool.shape[0] // PR, dtype=torch.int32).cuda(), torch.zeros(T, dtype=torch.int32).cuda(), torch.tensor(pos, dtype=torch.int32).cuda()]
    out = torch.empty(T, heads, W, device="cuda")
    a = S.LatentAttentionArgs()
    a.qa, a.out, a.pool, a.pages, a.max_pages, a.page_rows = dev[0].data_ptr(), out.data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), dev[2].numel(), PR
    a.slot, a.pos, a.scale = dev[3].data_ptr(), dev[4].data_ptr(), scale
    a.n_tokens, a.heads, a.rank, a.dtype, a.longest_entry, a.longest_context, a.out_cols = T, heads, W, S.BF16, 1, n, cols
    torch.cuda.synchronize()
    assert S.lib().b200_latent_attention_ex(C.byref(a), None) == 0
    torch.cuda.synchronize()
    kv = rows.double()
    s = qa.double() @ kv.T * scale
    s = s.masked_fill(torch.arange(n)[None, None, :] > torch.tensor(pos)[:, None, None], float("-inf"))
    want = torch.softmax(s, -1) @ kv[:, :cols]
    assert float((out.double().cpu()[:, :, :cols] - want).norm() / want.norm()) < 3e-5
