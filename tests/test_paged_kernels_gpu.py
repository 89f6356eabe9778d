"""The kernels behind b200_paged_attention in bfloat16, each over the sizes where its tiles end, against a plain float64 statement of
the attention (one sequence at a time, every option of the call)."""
import ctypes as C
import math

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


def seen(o, p):
    """first key that position p sees"""
    f = p // o["chunk"] * o["chunk"] if o.get("chunk") else 0
    return max(f, p - o["window"] + 1) if o.get("window") else f


def reference(q, k, v, pos, o):
    """q [T, H, M, d] at positions pos of ONE sequence with keys k [n, G, M, d], values v [n, G, dv] -> [T, H, M, dv]"""
    T, H, M, d = q.shape
    G, n = k.shape[1], k.shape[0]
    j, p = torch.arange(n), torch.tensor(pos)
    first = torch.tensor([seen(o, x) for x in pos])
    ok = (j[None, :] <= p[:, None]) & (j[None, :] >= first[:, None])
    out = torch.zeros(T, H, M, v.shape[2], dtype=torch.float64)
    for h in range(H):
        for m in range(M):
            s = q[:, h, m] @ k[:, h // (H // G), m].T * o["scale"]
            if o.get("cap"):
                s = o["cap"] * torch.tanh(s / o["cap"])
            if o.get("bias") is not None:
                s = s + o["bias"][h][(p[:, None] - j[None, :]).clamp(0, o["bias"].shape[1] - 1)]
            if o.get("sigmoid"):
                w = torch.sigmoid(s + o["head_bias"][h]) * ok
            else:
                s = s.masked_fill(~ok, float("-inf"))
                sink = o["sink"][h] if o.get("sink") is not None else torch.tensor(math.log(o["denom"]) if o.get("denom") else float("-inf"), dtype=torch.float64)
                top = torch.maximum(s.amax(1, keepdim=True), sink)
                e = torch.exp(s - top)
                w = e / (e.sum(1, keepdim=True) + torch.exp(sink - top))
            out[:, h, m] = w @ v[:, h // (H // G)]
    return out


def run(S, q, keys, values, table, PR, slot, pos, o, longest, f32=True, workspace=True):
    """one call over device tensors q [T, H, M, d] (bfloat16), pools [rows, G, M, d] / [rows, G, dv]"""
    T, H, M, d = q.shape
    G, dv = values.shape[1], values.shape[2]
    out = torch.full((T, H, M, dv), float("nan"), dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    keep = [torch.tensor(slot, dtype=torch.int32, device="cuda"), torch.tensor(pos, dtype=torch.int32, device="cuda")]
    a = S.PagedAttentionArgs()
    a.q, a.out, a.k_pool, a.v_pool, a.pages, a.max_pages, a.page_rows = q.data_ptr(), out.data_ptr(), keys.data_ptr(), values.data_ptr(), table.data_ptr(), table.shape[1], PR
    a.slot, a.pos, a.n_tokens, a.heads, a.kv_heads, a.dim, a.vdim = keep[0].data_ptr(), keep[1].data_ptr(), T, H, G, d, dv
    a.scale, a.softcap, a.denom_bias, a.dtype, a.longest_entry, a.longest_context = o["scale"], o.get("cap", 0.0), o.get("denom", 0.0), S.BF16, longest, max(pos) + 1
    a.chunk, a.maps, a.out_f32, a.window, a.sigmoid_weights = o.get("chunk", 0), M, int(f32), o.get("window", 0), int(bool(o.get("sigmoid")))
    for name, key in (("sink", "sink"), ("dist_bias", "bias"), ("head_bias", "head_bias"), ("head_temp", "temp")):
        if o.get(key) is not None:
            keep.append(o[key].float().cuda().contiguous())
            setattr(a, name, keep[-1].data_ptr())
    if o.get("bias") is not None:
        a.dist_n = o["bias"].shape[1]
    need = S.lib().b200_paged_attention_workspace_bytes(T, H * M, dv) if workspace else 0
    keep.append(torch.empty(max(need, 16), dtype=torch.uint8, device="cuda"))
    a.workspace, a.workspace_bytes = keep[-1].data_ptr(), need
    torch.cuda.synchronize()
    rc = S.lib().b200_paged_attention(C.byref(a), None)
    torch.cuda.synchronize()
    assert rc == 0, rc
    return out.double().cpu()


def sequences(g, lens, G, M, d, dv, PR):
    """keys and values per sequence, and pools in shuffled pages whose foreign rows are NaN: reading one would show"""
    k = [torch.randn(n, G, M, d, generator=g).bfloat16().double() for n in lens]
    v = [torch.randn(n, G, dv, generator=g).bfloat16().double() for n in lens]
    need = [(n + PR - 1) // PR for n in lens]
    order = torch.randperm(sum(need) + 2, generator=g).tolist()
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    kp = torch.full(((sum(need) + 2) * PR, G, M, d), float("nan"))
    vp = torch.full(((sum(need) + 2) * PR, G, dv), float("nan"))
    for b, n in enumerate(lens):
        for i in range(need[b]):
            pg, m = order.pop(), min(PR, n - i * PR)
            table[b, i] = pg
            kp[pg * PR:pg * PR + m], vp[pg * PR:pg * PR + m] = k[b][i * PR:i * PR + m], v[b][i * PR:i * PR + m]
    return k, v, kp.bfloat16().cuda(), vp.bfloat16().cuda(), table.cuda()


FORMS = {"plain": {}, "capped": dict(cap=3.0, denom=1.0), "biased": dict(sink=1, bias=40), "blocks": dict(chunk=100), "sigmoid": dict(window=70, sigmoid=1)}


def options(form, H, d, g):
    o = dict(FORMS[form], scale=1.3 / math.sqrt(d))
    if o.get("bias"):
        o["bias"], o["sink"] = torch.randn(H, o["bias"], generator=g).float().double(), torch.randn(H, generator=g).float().double() * 3
    if o.get("sigmoid"):
        o["head_bias"] = torch.randn(H, generator=g).float().double() - 2
    return o


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("H,G,M,d,dv,PR", [(2, 2, 1, 128, 128, 64), (8, 4, 1, 128, 128, 16), (6, 2, 1, 64, 64, 64), (8, 1, 1, 64, 128, 48), (4, 2, 2, 128, 256, 64)])
def test_single_tokens_share_their_context_in_a_cluster(S, form, H, G, M, d, dv, PR):
    """contexts that end at, before and behind a step of 16 keys, a page and a warp's share. The weights keep 24 bits, so the fp32
    output is as exact as fp32 sums of a thousand products: 2e-5 of the result's norm"""
    if M > 1 and FORMS[form].get("sigmoid"):
        pytest.skip("sigmoid weights have one map")
    g = torch.Generator().manual_seed(H * d + PR)
    lens = [1, 15, 16, 17, 63, 65, 300, 1100]
    o = options(form, H, d, g)
    k, v, kp, vp, table = sequences(g, lens, G, M, d, dv, PR)
    q = torch.randn(len(lens), H, M, d, generator=g).bfloat16().double()
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, list(range(len(lens))), [n - 1 for n in lens], o, 1)
    one = run(S, q[6:7].bfloat16().cuda(), kp, vp, table, PR, [6], [lens[6] - 1], o, 1, workspace=False)
    for b, n in enumerate(lens):
        want = reference(q[b:b + 1], k[b], v[b], [n - 1], o)[0]
        assert float((got[b] - want).norm() / want.norm()) < 2e-5, (b, n)
        if b == 6:
            assert float((one[0] - want).norm() / want.norm()) < 2e-5


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("H,G,M,d,dv,PR", [(2, 2, 1, 128, 128, 64), (8, 4, 1, 128, 128, 128), (6, 2, 1, 64, 64, 64), (8, 1, 1, 64, 64, 192), (4, 2, 2, 128, 256, 64)])
def test_prompt_portions_beside_single_tokens(S, form, H, G, M, d, dv, PR):
    """portions that end at, before and behind a tile of rows, contexts that end at, before and behind a tile of keys, several sequences
    in one window of rows, and single tokens between them. The weights are rounded to bfloat16 as operand of the second product: an
    independent error of at most 2^-9 in every weight, 1.2e-3 of the result's norm on average; 5e-3 is four times that"""
    if M > 1 and FORMS[form].get("sigmoid"):
        pytest.skip("sigmoid weights have one map")
    g = torch.Generator().manual_seed(H * d + PR + 1)
    o = options(form, H, d, g)
    before, new = [0, 250, 63, 3, 128, 0, 600, 64], [200, 1, 65, 2, 64, 129, 1, 1]
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], G, M, d, dv, PR)
    q = [torch.randn(n, H, M, d, generator=g).bfloat16().double() for n in new]
    for batch in (range(8), [0], [5, 2], [3, 4, 1], [7, 3], [2], [4]):
        batch = list(batch)
        slot = [b for b in batch for _ in range(new[b])]
        pos = [before[b] + i for b in batch for i in range(new[b])]
        got = run(S, torch.cat([q[b] for b in batch]).bfloat16().cuda(), kp, vp, table, PR, slot, pos, o, max(new[b] for b in batch), f32=batch != [0])
        at = 0
        for b in batch:
            want = reference(q[b], k[b], v[b], list(range(before[b], before[b] + new[b])), o)
            assert float((got[at:at + new[b]] - want).norm() / want.norm()) < 5e-3, (batch, b)
            at += new[b]


@pytest.mark.parametrize("R", [1, 2])
def test_weights_that_grow_along_the_keys(S, R):
    """scores that rise by hundreds from the first keys to the last: the running maximum has to be carried into what is already summed;
    and a head whose scale is negative"""
    g = torch.Generator().manual_seed(3)
    d, n, PR = 128, 520, 64
    k, v, kp, vp, table = sequences(g, [n], 1, 1, d, d, PR)
    ramp = torch.linspace(0.0, 6.0, n)[:, None, None, None].double()
    k = [(k[0] * 0.05 + ramp).bfloat16().double()]
    for i in range((n + PR - 1) // PR):
        m = min(PR, n - i * PR)
        pg = int(table[0, i])
        kp[pg * PR:pg * PR + m] = k[0][i * PR:i * PR + m].bfloat16().cuda()
    q = (torch.rand(n, R, 1, d, generator=g) + 0.2).bfloat16().double()
    for scale in (0.3, -0.3):
        got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * n, list(range(n)), dict(scale=scale), n)
        want = reference(q, k[0], v[0], list(range(n)), dict(scale=scale))
        assert float((got - want).norm() / want.norm()) < 5e-3, scale


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("H,G,M,d,dv", [(4, 2, 1, 128, 128), (6, 2, 1, 64, 64), (4, 2, 2, 128, 256)])
def test_prompt_weights_are_the_sum_of_two_bfloat16(S, form, H, G, M, d, dv):
    """fp32 outputs, more keys than the mma.sync tiles take. A weight keeps 16 bits (hi is cut off, lo rounded to 8 bits of what is left: off by at most 2^-16 of the weight, 2^-18 on average), the sums take 2 * 1280 / 16
    additions that are each off by at most 2^-23 (the tensor core truncates), the exponentials by 2^-22: 3e-5 in all. Weights rounded to bfloat16
    alone are off by 1e-3, and by more where a row's largest weight is not 1"""
    if M > 1 and FORMS[form].get("sigmoid"):
        pytest.skip("sigmoid weights have one map")
    g = torch.Generator().manual_seed(H * d + M)
    o = options(form, H, d, g)
    before, n, PR = 950, 330, 64
    k, v, kp, vp, table = sequences(g, [before + n], G, M, d, dv, PR)
    q = torch.randn(n, H, M, d, generator=g).bfloat16().double()
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * n, list(range(before, before + n)), o, n)
    want = reference(q, k[0], v[0], list(range(before, before + n)), o)
    assert float((got - want).norm() / want.norm()) < 3e-5


@pytest.mark.parametrize("form,before", [("blocks", 230), ("blocks", 305), ("sigmoid", 171)])
@pytest.mark.parametrize("d,dv", [(128, 128), (64, 64), (128, 256)])
def test_rows_ahead_of_the_first_visible_key_may_hold_anything(S, form, before, d, dv):
    """a portion whose window or block begins inside a page: what is cached ahead of it is NaN, as it is where only the visible part of a
    sequence was brought into the cache"""
    g = torch.Generator().manual_seed(before + dv)
    o = options(form, 4, d, g)
    n, PR = 70, 64
    k, v, kp, vp, table = sequences(g, [before + n], 2, 1, d, dv, PR)
    first = seen(o, before)
    for j in range(first):
        row = int(table[0, j // PR]) * PR + j % PR
        kp[row], vp[row] = float("nan"), float("nan")
    q = torch.randn(n, 4, 1, d, generator=g).bfloat16().double()
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * n, list(range(before, before + n)), o, n)
    want = reference(q, k[0], v[0], list(range(before, before + n)), o)
    assert float((got - want).norm() / want.norm()) < 3e-5


@pytest.mark.parametrize("G", [4, 2, 1])
@pytest.mark.parametrize("longest", [0, 1, 90])
def test_head_temperatures_and_an_unknown_longest_entry(S, G, longest):
    """a factor per head on the scores, negative ones among them; 0: the caller does not know how many tokens an entry brings"""
    g = torch.Generator().manual_seed(G + longest)
    H, d, PR = 4, 128, 64
    before, new = ([250, 63, 10], [1, 1, 1]) if longest == 1 else ([250, 63, 10, 0], [1, 65, 1, 90])
    o = dict(scale=1.3 / math.sqrt(d), temp=torch.tensor([0.5, -1.0, 1.7, 0.0], dtype=torch.float64))
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], G, 1, d, d, PR)
    q = [torch.randn(n, H, 1, d, generator=g).bfloat16().double() for n in new]
    slot = [b for b in range(len(new)) for _ in range(new[b])]
    pos = [before[b] + i for b in range(len(new)) for i in range(new[b])]
    got = run(S, torch.cat(q).bfloat16().cuda(), kp, vp, table, PR, slot, pos, o, longest)
    at = 0
    for b in range(len(new)):
        want = reference(q[b] * o["temp"][None, :, None, None], k[b], v[b], list(range(before[b], before[b] + new[b])), o)
        assert float((got[at:at + new[b]] - want).norm() / want.norm()) < 3e-5, b
        at += new[b]


@pytest.mark.parametrize("form", list(FORMS))
@pytest.mark.parametrize("H,G,M,d,dv", [(4, 2, 1, 128, 128), (6, 2, 1, 64, 64), (4, 2, 2, 128, 256)])
@pytest.mark.parametrize("before,new", [([760], [9]), ([1290], [70]), ([2110], [33]), ([2100, 0, 700, 5], [20, 40, 3, 1])])
def test_key_tiles_of_a_portion_are_shared_by_a_cluster(S, form, H, G, M, d, dv, before, new):
    """few rows behind long contexts: two, four and eight CTAs share the key tiles of a tile of rows; entries with fewer key tiles than CTAs, and a single token, beside them.
    fp32 outputs: the bound of test_prompt_weights_are_the_sum_of_two_bfloat16, whose chain of additions is longer"""
    if M > 1 and FORMS[form].get("sigmoid"):
        pytest.skip("sigmoid weights have one map")
    if d == 64 and form == "biased" and before == [760]:
        pytest.skip("up to 1200 keys these go to the mma.sync tiles, whose weights are rounded to bfloat16")
    g = torch.Generator().manual_seed(H * d + len(before))
    o = options(form, H, d, g)
    if o.get("chunk"):
        o["chunk"] = 1500
    if o.get("window"):
        o["window"] = 1100
    PR = 64
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], G, M, d, dv, PR)
    q = [torch.randn(n, H, M, d, generator=g).bfloat16().double() for n in new]
    slot = [b for b in range(len(new)) for _ in range(new[b])]
    pos = [before[b] + i for b in range(len(new)) for i in range(new[b])]
    got = run(S, torch.cat(q).bfloat16().cuda(), kp, vp, table, PR, slot, pos, o, max(new))
    at = 0
    for b in range(len(new)):
        want = reference(q[b], k[b], v[b], list(range(before[b], before[b] + new[b])), o)
        assert float((got[at:at + new[b]] - want).norm() / want.norm()) < 3e-5, b
        at += new[b]


@pytest.mark.parametrize("form", ["plain", "capped", "biased"])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("before", [[0, 130, 700, 40], [2100, 130, 700, 40]])
def test_more_tiles_than_the_gpu_holds_at_once(S, form, d, before):
    """several entries whose tiles come in more than one round: short contexts on two CTAs per SM, long ones sorted by what they see. The bound is that of portions beside single tokens"""
    g = torch.Generator().manual_seed(d + before[0])
    H, new, PR = 20, [130, 640, 500, 1], 64
    o = options(form, H, d, g)
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], H, 1, d, d, PR)
    q = [torch.randn(n, H, 1, d, generator=g).bfloat16().double() for n in new]
    slot = [b for b in range(4) for _ in range(new[b])]
    pos = [before[b] + i for b in range(4) for i in range(new[b])]
    got = run(S, torch.cat(q).bfloat16().cuda(), kp, vp, table, PR, slot, pos, o, max(new), f32=False)
    at = 0
    for b in range(4):
        want = reference(q[b], k[b], v[b], list(range(before[b], before[b] + new[b])), o)
        assert float((got[at:at + new[b]] - want).norm() / want.norm()) < 5e-3, b
        at += new[b]


@pytest.mark.parametrize("T", [1, 60, 80])
def test_precision_of_single_tokens_does_not_hang_on_the_shares(S, T):
    """fp32 outputs of 1500 keys in eight shares, two and one. A warp adds up to 24 steps in fp32, each rounded to 2^-24 of a sum that grows to 1: 24^0.5 / 3 * 2^-24 = 1.0e-7, and as
    much from a step's products and the exponentials; 4e-7 is twice both. Sums left to the tensor core are cut off three times a step: 24 * 3 * 2^-24 / 6 = 7e-7 for one share"""
    g = torch.Generator().manual_seed(T)
    H, d, n, PR = 2, 128, 1500, 64
    o = dict(options("sigmoid", H, d, g), window=0)
    k, v, kp, vp, table = sequences(g, [n], H, 1, d, d, PR)
    q = torch.randn(T, H, 1, d, generator=g).bfloat16().double()
    pos = [n - 1 - i for i in range(T)]
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * T, pos, o, 1)
    want = reference(q, k[0], v[0], pos, o)
    assert float((got - want).norm() / want.norm()) < 4e-7


@pytest.mark.parametrize("H,before,new", [(4, [250, 63, 10, 0], [1, 65, 1, 90]), (20, [2100, 130, 700, 40], [130, 640, 500, 1])])
@pytest.mark.parametrize("beyond", [1, 4000])
def test_a_limit_given_as_the_longest_entry(S, H, before, new, beyond):
    """a number that no entry can have is as good as none: the same kernels, so the same bits, single tokens behind the portions' tiles and ahead of them"""
    g = torch.Generator().manual_seed(H + beyond)
    d, PR = 128, 64
    o = options("plain", H, d, g)
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], H, 1, d, d, PR)
    q = torch.cat([torch.randn(n, H, 1, d, generator=g).bfloat16() for n in new])
    slot = [b for b in range(len(new)) for _ in range(new[b])]
    pos = [before[b] + i for b in range(len(new)) for i in range(new[b])]
    unknown, limit = (run(S, q.cuda(), kp, vp, table, PR, slot, pos, o, longest) for longest in (0, len(pos) + beyond))
    assert torch.equal(unknown, limit)
    at = 0
    for b in range(len(new)):
        want = reference(q[at:at + new[b]].double(), k[b], v[b], list(range(before[b], before[b] + new[b])), o)
        assert float((limit[at:at + new[b]] - want).norm() / want.norm()) < 3e-5, b   # (the bound of fp32 outputs of portions)
        at += new[b]


@pytest.mark.parametrize("form", ["plain", "biased", "sigmoid"])
@pytest.mark.parametrize("T,PR", [(1, 16), (9, 80), (25, 64), (40, 16)])
def test_single_tokens_of_narrow_heads(S, form, T, PR):
    """heads of 64 / 64, whose rows come by copies of 16 bytes: eight shares of a context to one, runs of steps shorter and longer than the ring, up to four CTAs per SM, contexts that begin
    and end inside a step. The bound of test_single_tokens_share_their_context_in_a_cluster"""
    g = torch.Generator().manual_seed(T + PR)
    H, d, n = 8, 64, 1101
    o = options(form, H, d, g)
    k, v, kp, vp, table = sequences(g, [n], H, 1, d, d, PR)
    q = torch.randn(T, H, 1, d, generator=g).bfloat16().double()
    pos = [n - 1 - 27 * i for i in range(T)]
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * T, pos, o, 1)
    want = reference(q, k[0], v[0], pos, o)
    assert float((got - want).norm() / want.norm()) < 2e-5


@pytest.mark.parametrize("H,before,new", [(4, [250, 63, 10, 0], [1, 65, 1, 90]), (16, [2100, 130, 700, 40, 1900], [130, 400, 1, 1, 1]), (8, [700, 2000, 40], [1, 1, 1]), (8, [300], [500])])
def test_inputs_rewritten_by_the_kernels_ahead(S, H, before, new):
    """queries and keys are rewritten by the library's own kernels, launched programmatically directly ahead of each call, several times in one stream: the bits of the same calls with the
    GPU waited for in between. A kernel that read ahead of what it depends on, or lines that it still held, would show"""
    g = torch.Generator().manual_seed(H + len(new))
    d, PR, rounds = 128, 64, 6
    lib, T = S.lib(), sum(new)
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], H, 1, d, d, PR)
    vp.nan_to_num_(0.0)
    slot = torch.tensor([b for b in range(len(new)) for _ in range(new[b])], dtype=torch.int32).cuda()
    pos = torch.tensor([before[b] + i for b in range(len(new)) for i in range(new[b])], dtype=torch.int32).cuda()
    W, rows, q = H * d, kp.shape[0], torch.empty(T, H * d, dtype=torch.bfloat16, device="cuda")
    one, zero = torch.ones(W, device="cuda"), torch.zeros(W, device="cuda")
    src = [[torch.randn(n, W, generator=g).cuda() for n in (T, rows)] for _ in range(rounds)]
    outs = [[torch.zeros(T, W, dtype=torch.float32, device="cuda") for _ in range(rounds)] for _ in range(2)]
    a = S.PagedAttentionArgs()
    a.q, a.k_pool, a.v_pool, a.pages, a.max_pages, a.page_rows = q.data_ptr(), kp.data_ptr(), vp.data_ptr(), table.data_ptr(), table.shape[1], PR
    a.slot, a.pos, a.n_tokens, a.heads, a.kv_heads, a.dim, a.vdim, a.scale = slot.data_ptr(), pos.data_ptr(), T, H, H, d, d, d ** -0.5
    a.dtype, a.longest_entry, a.longest_context, a.out_f32 = S.BF16, max(new), max(x + y for x, y in zip(before, new)), 1
    for waited in (0, 1):
        work = [[t.clone() for t in s] for s in src]   # (the norm adds to its input in place)
        torch.cuda.synchronize()
        for i in range(rounds):
            for x, n, to in ((work[i][0], T, q), (work[i][1], rows, kp)):
                assert lib.b200_layernorm_residual(x.data_ptr(), src[i][0 if n == T else 1].data_ptr(), n, W, 1e-5, 0.5, one.data_ptr(), zero.data_ptr(), one.data_ptr(), zero.data_ptr(), to.data_ptr(), S.BF16, None) == 0
                if waited:
                    torch.cuda.synchronize()
            a.out = outs[waited][i].data_ptr()
            assert lib.b200_paged_attention(C.byref(a), None) == 0
            if waited:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
    for i in range(rounds):
        assert torch.equal(outs[0][i], outs[1][i]), i
        assert bool(outs[0][i].isfinite().all()) and (i == 0 or not torch.equal(outs[0][i], outs[0][i - 1])), i


@pytest.mark.parametrize("H,d,dv", [(8, 128, 128), (8, 64, 128), (8, 128, 256)])
def test_three_shares_of_a_context(S, H, d, dv):
    """just more (token, key head) pairs than SMs behind more than 1200 keys: clusters of three, whose parts of the outputs do not come out even. The bound of
    test_single_tokens_share_their_context_in_a_cluster"""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator().manual_seed(d + dv)
    T, n, PR, o = sms // H + 1, 1301, 64, options("plain", H, d, g)
    k, v, kp, vp, table = sequences(g, [n], H, 1, d, dv, PR)
    q = torch.randn(T, H, 1, d, generator=g).bfloat16().double()
    pos = [n - 1 - 61 * i for i in range(T)]
    got = run(S, q.bfloat16().cuda(), kp, vp, table, PR, [0] * T, pos, o, 1)
    want = reference(q, k[0], v[0], pos, o)
    assert float((got - want).norm() / want.norm()) < 2e-5


@pytest.mark.parametrize("before", [[0, 130, 700, 40], [2100, 130, 700, 40]])
def test_more_tiles_of_wide_values_than_the_gpu_holds_at_once(S, before):
    """values of 256 columns, whose tiles take an SM alone: the bound of test_more_tiles_than_the_gpu_holds_at_once"""
    g = torch.Generator().manual_seed(before[0] + 256)
    H, d, new, PR = 20, 128, [130, 640, 500, 1], 64
    o = options("capped", H, d, g)
    k, v, kp, vp, table = sequences(g, [a + b for a, b in zip(before, new)], H, 1, d, 256, PR)
    q = [torch.randn(n, H, 1, d, generator=g).bfloat16().double() for n in new]
    slot = [b for b in range(4) for _ in range(new[b])]
    pos = [before[b] + i for b in range(4) for i in range(new[b])]
    got = run(S, torch.cat(q).bfloat16().cuda(), kp, vp, table, PR, slot, pos, o, max(new), f32=False)
    at = 0
    for b in range(4):
        want = reference(q[b], k[b], v[b], list(range(before[b], before[b] + new[b])), o)
        assert float((got[at:at + new[b]] - want).norm() / want.norm()) < 5e-3, b
        at += new[b]


@pytest.mark.parametrize("form,before,n", [("plain", 0, 1300), ("plain", 1500, 500), ("blocks", 0, 1300), ("sigmoid", 0, 1300), ("biased", 0, 1300), ("capped", 0, 1300)])
@pytest.mark.parametrize("H,G,d", [(32, 16, 128), (32, 8, 64)])
def test_one_prompt_of_more_tiles_than_two_rounds(S, form, before, n, H, G, d):
    """one entry whose tiles come in more than two rounds, or behind more than it brings in more than one: one group of softmax warps and two CTAs per SM, where staged bias numbers leave room for
    them. The bound of test_prompt_portions_beside_single_tokens"""
    g = torch.Generator().manual_seed(H + before + d)
    o = options(form, H, d, g)
    if o.get("window"):
        o["window"] = 500
    k, v, kp, vp, table = sequences(g, [before + n], G, 1, d, d, 64)
    q = torch.randn(n, H, 1, d, generator=g).bfloat16().double()
    pos = list(range(before, before + n))
    got = run(S, q.bfloat16().cuda(), kp, vp, table, 64, [0] * n, pos, o, n, f32=False)
    want = reference(q, k[0], v[0], pos, o)
    assert float((got - want).norm() / want.norm()) < 5e-3
