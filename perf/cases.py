"""Cases that stand for what users of this framework run, for timing and for comparing one version's outputs with another's.

The serving layer (`include/b200_serve.h`) runs any mix of prompt portions and single decoded tokens as one batch, in bfloat16 with
fp32 accumulation; its layers are attention over paged keys and values, latent attention over paged low-rank rows, dense and routed
feed-forwards, and recurrences with a state per sequence. Each of them is called here as a family's step calls it, at the sizes of the
configurations in `llm-inference_b200/bench_families.py` (size m unless a case says otherwise) and at odd sizes around them. Two cases are whole calls:
a Musilorn model through `b200_model_step`, and the LLaMA-2-7B-shaped engine of `include/b200_engine.h` in fp16.

A case is a dict of plain values; lengths of ragged batches follow from it, values from the seed.
"""
import ctypes as C
import math
import tempfile

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()
S, E, capi = pkg.serve, pkg.engine, pkg.capi
PAGE = 64   # rows of a cache page, as every family of the serving layer allocates them
GOLDEN = 0.6180339887498949


def listed():
    return [
        # one user's chat: a single sequence decodes its next token (size s); the smallest call, launches and latency
        dict(name="attention_decode_one", op="attention", portions=0, portion=0, singles=1, context=500, heads=8, kv_heads=4, dim=128, form="plain"),
        # a serving batch decodes: 32 ragged sequences, Mazotar's attention (distance bias, learned sinks)
        dict(name="attention_decode_batch", op="attention", portions=0, portion=0, singles=32, context=2048, heads=16, kv_heads=8, dim=128, form="biased"),
        # a prompt is read at once (Tomalix' plain attention)
        dict(name="attention_prompt", op="attention", portions=1, portion=2048, singles=0, context=0, heads=16, kv_heads=8, dim=128, form="plain"),
        # continuous batching: three prompts in portions of 512 behind what they have cached, beside twelve decoding sequences (Musilorn's attention)
        dict(name="attention_mixed", op="attention", portions=3, portion=512, singles=12, context=4000, heads=16, kv_heads=8, dim=128, form="capped"),
        # latent attention with a rotated key part (Filipel, Sakevik): a decode batch, and a whole prompt
        dict(name="latent_decode", op="latent", portions=0, portion=0, singles=8, context=1024, heads=16, rank=512, extra=64, sink=False, window=0),
        dict(name="latent_prompt", op="latent", portions=1, portion=2048, singles=0, context=0, heads=16, rank=512, extra=64, sink=False, window=0),
        # the query / key / value projection of eight decoding sequences; the gated feed-forward of a 2048-token prompt
        dict(name="linear_decode", op="linear", rows=8, k=2048, n=4096, epi="none"),
        dict(name="linear_prompt", op="linear", rows=2048, k=2048, n=5504, epi="glu"),
        # routed experts (Nekodra) for a prompt portion of 512 tokens: dispatch, gated products, down products, residual
        dict(name="experts_portion", op="experts", rows=512, width=2048, ff=1024, experts=16, top=4),
        # the state-space recurrence of Filipel over two prompts
        dict(name="recurrence_prompt", op="recurrence", entries=2, tokens=2048, heads=64, vdim=64, n_state=128),
        # four requests through a whole Musilorn model (size s): prompts in one step, then four decode steps
        dict(name="model_serve", op="model", requests=4, prompt=512, steps=4),
        # two LLaMA-2-7B-shaped layers with embedding and head, fp16: a 512-token prompt, then four decode steps
        dict(name="llama_serve", op="llama", batch=1, prompt=512, steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["attention", "attention", "attention", "latent", "latent", "linear", "linear", "experts", "recurrence", "model", "llama"])
    if op == "attention":
        heads, kv = rng.choice([(16, 8), (16, 8), (8, 4), (16, 4), (16, 16)])
        c = dict(op=op, heads=heads, kv_heads=kv, dim=rng.choice([128, 128, 128, 64]), form=rng.choice(["plain", "capped", "biased", "sigmoid", "blocks"]))
        kind = rng.choice(["decode", "prompt", "mixed"])
        if kind == "decode":
            return dict(c, portions=0, portion=0, singles=_log(rng, 1, 32), context=_log(rng, 60, 2048))
        if kind == "prompt":
            n = rng.randint(1, 3)
            return dict(c, portions=n, portion=_log(rng, 40, 2048 // n), singles=0, context=0)
        return dict(c, portions=rng.randint(1, 3), portion=_log(rng, 16, 512), singles=rng.randint(1, 12), context=_log(rng, 100, 4000))
    if op == "latent":
        rank, extra = rng.choice([(512, 64), (512, 64), (512, 0), (256, 64)])
        c = dict(op=op, heads=16 if rank == 512 else 8, rank=rank, extra=extra, sink=extra == 0, window=rng.choice([0, 0, 1024]))
        if rng.random() < 0.5:
            return dict(c, portions=0, portion=0, singles=_log(rng, 1, 32), context=_log(rng, 60, 2048))
        n = rng.randint(1, 3)
        return dict(c, portions=n, portion=_log(rng, 40, 2048 // n), singles=rng.choice([0, 3]), context=rng.choice([0, _log(rng, 60, 1000)]) if n > 1 else 0)
    if op == "linear":
        n, k = rng.choice([(4096, 2048), (2048, 2048), (2048, 5504), (2048, 8192), (3072, 1024), (1024, 2688), (2048, 1408), (1000, 1032), (6184, 2048)])
        epi = rng.choice(["none", "none", "glu", "relu2"])
        if epi == "glu":
            n, k = rng.choice([(5504, 2048), (8192, 2048), (2688, 1024), (4096, 1024)])
        return dict(op=op, rows=_log(rng, 1, 2048 * 5504 // max(n, 5504)), k=k, n=n, epi=epi)
    if op == "experts":
        width, ff, experts, top = rng.choice([(2048, 1024, 16, 4), (1024, 512, 8, 2), (2048, 1408, 16, 3), (1024, 640, 16, 4)])
        return dict(op=op, rows=_log(rng, 1, 512), width=width, ff=ff, experts=experts, top=top)
    if op == "recurrence":
        heads, n_state = rng.choice([(64, 128), (32, 128), (64, 64), (33, 128)])
        return dict(op=op, entries=rng.randint(1, 4), tokens=_log(rng, 560, 2048), heads=heads, vdim=64, n_state=n_state)
    if op == "model":
        return dict(op=op, requests=rng.randint(1, 4), prompt=_log(rng, 20, 500), steps=rng.randint(1, 4))
    return dict(op=op, batch=rng.choice([1, 1, 2]), prompt=_log(rng, 16, 240), steps=rng.randint(1, 4))


# ---- inputs ------------------------------------------------------------------------------------------------------
def _lengths(n, most):
    """n ragged lengths up to `most`, the first the longest"""
    return [max(1, int(most * (1 - 0.6 * ((i * GOLDEN) % 1.0)))) for i in range(n)]


def _entries(c):
    """(cached rows, new tokens) of every sequence of a batch: prompt portions, then single tokens"""
    sizes, before = _lengths(c["portions"], c["portion"]), _lengths(c["portions"], c["context"]) if c["context"] else [0] * c["portions"]
    return list(zip(before, sizes)) + [(n, 1) for n in _lengths(c["singles"], c["context"])]


def _seen(c, p):
    """first key that position p sees"""
    if c.get("window"):
        return max(0, p - c["window"] + 1)
    if c.get("form") == "sigmoid":
        return max(0, p - 1023)
    return p // 1024 * 1024 if c.get("form") == "blocks" else 0


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rnd(g, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _f64(t):
    return t.to(torch.float64)


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _ok(rc):
    if rc != 0:
        raise RuntimeError("rc=%d" % rc)


def _pages(ent, g):
    """a shuffled page list per sequence: (table on the GPU, rows of the pool, pool row of every cached row per sequence)"""
    need = [(a + n + PAGE - 1) // PAGE for a, n in ent]
    total, most = sum(need), max(need)
    order = torch.randperm(total, generator=g, device="cuda").to(torch.int32)
    table, rows, at = torch.zeros(len(ent), most, dtype=torch.int32, device="cuda"), [], 0
    for b, n in enumerate(need):
        table[b, :n] = order[at:at + n]
        rows.append((order[at:at + n].long()[:, None] * PAGE + torch.arange(PAGE, device="cuda")[None, :]).reshape(-1)[:sum(ent[b])])
        at += n
    return table, total * PAGE, rows


def _batch(ent):
    slot = [b for b, (_, n) in enumerate(ent) for _ in range(n)]
    pos = [a + i for a, n in ent for i in range(n)]
    return _i32(slot), _i32(pos), len(slot)


def _attention_inputs(c, seed):
    g, ent = _gen(seed), _entries(c)
    table, n_rows, rows = _pages(ent, g)
    slot, pos, T = _batch(ent)
    H, G, d = c["heads"], c["kv_heads"], c["dim"]
    bf = torch.bfloat16
    t = dict(q=_rnd(g, T, H * d, dtype=bf), k=_rnd(g, n_rows, G, d, dtype=bf), v=_rnd(g, n_rows, G, d, dtype=bf), table=table, slot=slot, pos=pos)
    t["bias"] = _rnd(g, H, 600, std=0.5)
    t["sink"], t["head_bias"] = _rnd(g, H), _rnd(g, H) - 5.0
    return t, ent, rows, T


def _latent_inputs(c, seed):
    g, ent = _gen(seed), _entries(c)
    table, n_rows, rows = _pages(ent, g)
    slot, pos, T = _batch(ent)
    W = c["rank"] + c["extra"]
    qa = _rnd(g, T, c["heads"], W, std=0.5)
    return dict(qa=qa, pool=_rnd(g, n_rows, W, dtype=torch.bfloat16), sink=_rnd(g, c["heads"]), table=table, slot=slot, pos=pos), ent, rows, T


def _linear_inputs(c, seed):
    g = _gen(seed)
    n_w = c["n"] * (2 if c["epi"] == "glu" else 1)
    return dict(x=_rnd(g, c["rows"], c["k"], dtype=torch.bfloat16), w=_rnd(g, n_w, c["k"], std=c["k"] ** -0.5, dtype=torch.bfloat16))


def _expert_inputs(c, seed):
    g = _gen(seed)
    T, D, F, X, k = c["rows"], c["width"], c["ff"], c["experts"], c["top"]
    score = torch.rand(T, X, generator=g, device="cuda") + 0.3 * torch.rand(1, X, generator=g, device="cuda")   # some experts are liked more
    w, chosen = torch.topk(score, k, dim=1)
    return dict(h=_rnd(g, T, D, dtype=torch.bfloat16), up=_rnd(g, X, 2 * F, D, std=D ** -0.5, dtype=torch.bfloat16),
                down=_rnd(g, X, D, F, std=F ** -0.5, dtype=torch.bfloat16), chosen=chosen.to(torch.int32).contiguous(),
                weight=(w / w.sum(1, keepdim=True)).contiguous(), x=_rnd(g, T, D, std=0.05))


def _recurrence_entries(c):
    share = _lengths(c["entries"], 1000)
    sizes = [max(1, c["tokens"] * s // sum(share)) for s in share]
    return [c["tokens"] - sum(sizes[1:])] + sizes[1:]


def _recurrence_inputs(c, seed):
    g, T, H, N, P = _gen(seed), c["tokens"], c["heads"], c["n_state"], c["vdim"]
    A = -torch.exp(torch.rand(H, generator=g, device="cuda") * math.log(16.0))
    return dict(u=_rnd(g, T, H * P + 2 * N, std=0.7), dt=_rnd(g, T, H), dt_bias=_rnd(g, H, std=0.5) - 3.0, A=A, D=torch.ones(H, device="cuda"))


MODEL = dict(vocab=32000, width=1024, heads=8, kv_heads=4, dim=128, ff=4096, taps=4, ret_heads=4, ret_dim=128, ret_vdim=256, layers=4)
LLAMA = dict(layers=2, heads=32, dim=128, inter=11008, vocab=32000)


def _model_weights(seed):
    m, g = MODEL, _gen(seed)
    D = m["width"]

    def mat(*shape, std=None):
        return _rnd(g, *shape, std=shape[-1] ** -0.5 if std is None else std, dtype=torch.bfloat16)

    def vec(n):
        return (1 + _rnd(g, n, std=0.05)).to(torch.bfloat16), _rnd(g, n, std=0.02, dtype=torch.bfloat16)

    w = {"embed": mat(m["vocab"], D, std=1.0), "head": mat(m["vocab"], D)}
    w["final.norm"], w["final.norm.b"] = vec(D)
    cfg = dict(architecture="Musilorn", vocab=m["vocab"], width=D, norm=dict(eps=1e-5), residual_mult=0.5, logit_softcap=25.0, layers=[])
    for i in range(m["layers"]):
        pre, last = "l%d." % i, i == m["layers"] - 1
        for name in ("norm1", "norm1b") + (() if last else ("norm2", "norm2b")):
            w[pre + name], w[pre + name + ".b"] = vec(D)
        if last:
            H, d, dv = m["ret_heads"], m["ret_dim"], m["ret_vdim"]
            for name, n in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv)):
                w[pre + "mix." + name] = mat(n, D)
            w[pre + "mix.o"] = mat(D, H * dv)
            cfg["layers"].append(dict(type="retention", mlp=None, mixer=dict(heads=H, dim=d, vdim=dv, rot=dict(base=10000.0, dims=d),
                                                                             decay=[1 - 2.0 ** (-5 - 5 * h / (H - 1)) for h in range(H)])))
            continue
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        w[pre + "mix.q"], w[pre + "mix.k"], w[pre + "mix.o"] = mat(H * d, D), mat(G * d, D), mat(D, H * d)
        w[pre + "mix.q.conv"], w[pre + "mix.k.conv"] = mat(H * d, m["taps"], std=0.5), mat(G * d, m["taps"], std=0.5)
        w[pre + "mix.q.norm"], w[pre + "mix.k.norm"] = vec(d)[0], vec(d)[0]
        w[pre + "mlp.gate"], w[pre + "mlp.up"], w[pre + "mlp.down"] = mat(m["ff"], D), mat(m["ff"], D), mat(D, m["ff"])
        cfg["layers"].append(dict(type="attention", mlp=dict(kind="dense", ff=m["ff"]),
                                  mixer=dict(heads=H, kv_heads=G, dim=d, vdim=d, conv=m["taps"], scale=d ** -0.5, softcap=50.0,
                                             rot=dict(base=500000.0, dims=d))))
    return cfg, w


def _tokens(vocab, n, seed):
    return np.random.default_rng(int(seed)).integers(0, vocab, n).astype(np.int32)


def _model_tokens(c, seed):
    return [_tokens(MODEL["vocab"], n + c["steps"], seed * 64 + i).tolist() for i, n in enumerate(_lengths(c["requests"], c["prompt"]))]


def _llama_weights(seed):
    m, g, out = LLAMA, _gen(seed), []
    H = m["heads"] * m["dim"]
    shapes = {E.W_QKV: (3 * H, H), E.W_O: (H, H), E.W_GATE_UP: (2 * m["inter"], H), E.W_DOWN: (H, m["inter"])}
    for layer in range(m["layers"]):
        out += [(E.W_ATTN_NORM, layer, 1 + _rnd(g, H, std=0.05)), (E.W_FFN_NORM, layer, 1 + _rnd(g, H, std=0.05))]
        out += [(slot, layer, _rnd(g, *s, std=s[1] ** -0.5)) for slot, s in shapes.items()]
    out += [(E.W_EMBED, 0, _rnd(g, m["vocab"], H)), (E.W_FINAL_NORM, 0, 1 + _rnd(g, H, std=0.05)), (E.W_LM_HEAD, 0, _rnd(g, m["vocab"], H, std=H ** -0.5))]
    return [(slot, layer, t.to(torch.float16)) for slot, layer, t in out]


def _llama_tokens(c, seed):
    return _tokens(LLAMA["vocab"], c["batch"] * (c["prompt"] + c["steps"]), seed).reshape(c["batch"], -1)


# ---- the calls ---------------------------------------------------------------------------------------------------
def prepare(c, seed):
    L = S.lib()
    if c["op"] == "attention":
        t, ent, _, T = _attention_inputs(c, seed)
        f32 = c["form"] in ("sigmoid", "blocks")   # layers whose heads are gated afterwards take fp32
        t["out"] = torch.empty(T, c["heads"] * c["dim"], dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
        need = L.b200_paged_attention_workspace_bytes(T, c["heads"], c["dim"])
        t["ws"] = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        a = S.PagedAttentionArgs()
        a.q, a.out, a.k_pool, a.v_pool = t["q"].data_ptr(), t["out"].data_ptr(), t["k"].data_ptr(), t["v"].data_ptr()
        a.pages, a.max_pages, a.page_rows, a.slot, a.pos = t["table"].data_ptr(), t["table"].shape[1], PAGE, t["slot"].data_ptr(), t["pos"].data_ptr()
        a.n_tokens, a.heads, a.kv_heads, a.dim, a.vdim, a.scale, a.dtype = T, c["heads"], c["kv_heads"], c["dim"], c["dim"], c["dim"] ** -0.5, S.BF16
        a.longest_entry, a.longest_context, a.out_f32 = max(n for _, n in ent), max(sum(e) for e in ent), int(f32)
        a.workspace, a.workspace_bytes = t["ws"].data_ptr(), need
        if c["form"] == "capped":
            a.softcap, a.denom_bias = 50.0, 1.0
        elif c["form"] == "biased":
            a.sink, a.dist_bias, a.dist_n = t["sink"].data_ptr(), t["bias"].data_ptr(), t["bias"].shape[1]
        elif c["form"] == "sigmoid":
            a.window, a.sigmoid_weights, a.head_bias = 1024, 1, t["head_bias"].data_ptr()
        elif c["form"] == "blocks":
            a.chunk = 1024
        return dict(op="attention", t=t, a=a, lib=L)
    if c["op"] == "latent":
        t, ent, _, T = _latent_inputs(c, seed)
        W = c["rank"] + c["extra"]
        t["out"] = torch.zeros(T, c["heads"], W, device="cuda")
        need = L.b200_latent_attention_workspace_bytes(T, c["heads"], W)
        t["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda")
        a = S.LatentAttentionArgs()
        a.qa, a.out, a.pool, a.pages, a.max_pages, a.page_rows = t["qa"].data_ptr(), t["out"].data_ptr(), t["pool"].data_ptr(), t["table"].data_ptr(), t["table"].shape[1], PAGE
        a.slot, a.pos, a.sink = t["slot"].data_ptr(), t["pos"].data_ptr(), t["sink"].data_ptr() if c["sink"] else None
        a.scale, a.n_tokens, a.heads, a.rank, a.window, a.dtype = 192 ** -0.5, T, c["heads"], W, c["window"], S.BF16
        a.longest_entry, a.longest_context, a.out_cols = max(n for _, n in ent), max(sum(e) for e in ent), c["rank"]
        a.workspace, a.workspace_bytes = t["ws"].data_ptr(), need
        return dict(op="latent", t=t, a=a, lib=L, cols=c["rank"])
    if c["op"] == "linear":
        t = _linear_inputs(c, seed)
        f32 = c["epi"] == "none"   # projections leave as fp32, activations as bfloat16: the next product's operand
        t["y"] = torch.empty(c["rows"], c["n"], dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
        need = L.b200_linear_ex_workspace_bytes(c["rows"], c["n"], c["k"])
        t["ws"] = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        epi = dict(none=S.GG_NONE, glu=S.GG_GLU, relu2=S.GG_RELU2)[c["epi"]]
        args = (t["x"].data_ptr(), t["w"].data_ptr(), t["y"].data_ptr(), c["rows"], c["n"], c["k"], S.BF16, S.F32 if f32 else S.BF16, epi, t["ws"].data_ptr(), need)
        return dict(op="linear", t=t, args=args, lib=L)
    if c["op"] == "experts":
        t = _expert_inputs(c, seed)
        T, D, F, X, k = c["rows"], c["width"], c["ff"], c["experts"], c["top"]
        t.update(off=torch.zeros(X + 1, dtype=torch.int32, device="cuda"), src=torch.zeros(T * k, dtype=torch.int32, device="cuda"),
                 dest=torch.zeros(T, k, dtype=torch.int32, device="cuda"), act=torch.zeros(T * k, F, dtype=torch.bfloat16, device="cuda"),
                 eo=torch.zeros(T * k, D, device="cuda"))
        up, down = S.GemmGroupedArgs(), S.GemmGroupedArgs()
        up.A, up.lda, up.a_rows, up.group_off, up.W, up.ldw, up.stride_w = t["h"].data_ptr(), D, t["src"].data_ptr(), t["off"].data_ptr(), t["up"].data_ptr(), D, 2 * F * D
        up.C, up.ldc, up.M, up.N, up.K, up.batch, up.trans_b, up.epi = t["act"].data_ptr(), F, T, F, D, X, 1, S.GG_GLU
        up.a_dtype = up.w_dtype = up.c_dtype = S.BF16
        down.A, down.lda, down.group_off, down.W, down.ldw, down.stride_w = t["act"].data_ptr(), F, t["off"].data_ptr(), t["down"].data_ptr(), F, D * F
        down.C, down.ldc, down.M, down.N, down.K, down.batch, down.trans_b, down.epi = t["eo"].data_ptr(), D, T, D, F, X, 1, S.GG_NONE
        down.a_dtype, down.w_dtype, down.c_dtype = S.BF16, S.BF16, S.F32
        return dict(op="experts", t=t, c=c, up=up, down=down, lib=L)
    if c["op"] == "recurrence":
        t, sizes = _recurrence_inputs(c, seed), _recurrence_entries(c)
        T, H, N, P = c["tokens"], c["heads"], c["n_state"], c["vdim"]
        rows = [sum(sizes[:i]) for i in range(len(sizes))]
        t.update(state=torch.zeros(len(sizes), H, N, P, device="cuda"), out=torch.empty(T, H * P, device="cuda"), ent_row=_i32(rows), ent_len=_i32(sizes),
                 slot=_i32([e for e, n in enumerate(sizes) for _ in range(n)]), pos=_i32([i for n in sizes for i in range(n)]))
        need = L.b200_ssd_scan_workspace_bytes(T, len(sizes), H, 1, P, N)
        t["ws"] = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        a = S.SsdScanArgs()
        a.u, a.ld_u, a.x_off, a.b_off, a.c_off = t["u"].data_ptr(), H * P + 2 * N, 0, H * P, H * P + N
        a.dt_raw, a.ld_dt, a.dt_bias, a.A, a.D = t["dt"].data_ptr(), H, t["dt_bias"].data_ptr(), t["A"].data_ptr(), t["D"].data_ptr()
        a.state, a.out, a.ent_row, a.ent_len, a.slot, a.pos = (t[n].data_ptr() for n in ("state", "out", "ent_row", "ent_len", "slot", "pos"))
        a.n_entries, a.n_tokens, a.heads, a.groups, a.vdim, a.n_state, a.longest_entry, a.chunked = len(sizes), T, H, 1, P, N, max(sizes), 1
        a.workspace, a.workspace_bytes = t["ws"].data_ptr(), need
        return dict(op="recurrence", t=t, a=a, lib=L)
    if c["op"] == "model":
        cfg, w = _model_weights(seed)
        seqs = _model_tokens(c, seed)
        with tempfile.TemporaryDirectory() as folder:
            S.write_checkpoint(folder, cfg, {k: v.cpu() for k, v in w.items()})
            model = S.Model(folder, dtype=S.BF16, max_tokens=sum(len(s) + PAGE for s in seqs), max_slots=len(seqs))
        return dict(op="model", model=model, seqs=seqs, steps=c["steps"])
    m = LLAMA
    eng = E.Engine(c["batch"], c["prompt"] + c["steps"] + 8, dtype=capi.F16, num_layers=m["layers"], head_num=m["heads"], kv_head_num=m["heads"],
                   head_size=m["dim"], inter_size=m["inter"], vocab_size=m["vocab"])
    for slot, layer, w in _llama_weights(seed):
        eng.weight_view(slot, layer).copy_(w)
    torch.cuda.synchronize()
    return dict(op="llama", eng=eng, ids=_llama_tokens(c, seed), prompt=c["prompt"], steps=c["steps"], stream=torch.cuda.ExternalStream(eng.stream))


def run(s):
    op = s["op"]
    if op == "attention":
        _ok(s["lib"].b200_paged_attention(C.byref(s["a"]), _stream()))
        return s["t"]["out"]
    if op == "latent":
        _ok(s["lib"].b200_latent_attention_ex(C.byref(s["a"]), _stream()))
        return s["t"]["out"][:, :, :s["cols"]]
    if op == "linear":
        _ok(s["lib"].b200_linear_ex(*s["args"], _stream()))
        return s["t"]["y"]
    if op == "experts":
        t, c, st = s["t"], s["c"], _stream()
        _ok(s["lib"].b200_moe_dispatch(t["chosen"].data_ptr(), c["rows"], c["top"], c["experts"], t["off"].data_ptr(), t["src"].data_ptr(), t["dest"].data_ptr(), st))
        _ok(s["lib"].b200_gemm_grouped(C.byref(s["up"]), st))
        _ok(s["lib"].b200_gemm_grouped(C.byref(s["down"]), st))
        _ok(s["lib"].b200_residual_combine(t["x"].data_ptr(), None, None, t["eo"].data_ptr(), t["dest"].data_ptr(), t["weight"].data_ptr(), t["h"].data_ptr(), S.BF16,
                                           c["rows"], c["width"], c["top"], st))
        return t["x"]
    if op == "recurrence":
        _ok(s["lib"].b200_ssd_scan(C.byref(s["a"]), _stream()))
        return [s["t"]["out"], s["t"]["state"]]
    if op == "model":
        m, out = s["model"], []
        for slot in range(len(s["seqs"])):
            m.release(slot)
        out.append(m.step([(b, q[:len(q) - s["steps"]], [len(q) - s["steps"] - 1]) for b, q in enumerate(s["seqs"])]))
        for i in range(s["steps"]):
            out.append(m.step([(b, [q[len(q) - s["steps"] + i]], [0]) for b, q in enumerate(s["seqs"])]))
        return out
    eng, out = s["eng"], []
    eng.reset()
    eng.prefill(s["ids"][:, :s["prompt"]])
    with torch.cuda.stream(s["stream"]):
        out.append(eng.logits().clone())
        for i in range(s["steps"]):
            eng.decode_step_host(s["ids"][:, s["prompt"] + i])
            out.append(eng.logits().clone())
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def work(c):
    if c["op"] == "attention":
        ent, d = _entries(c), c["dim"]
        pairs = sum(a + i + 1 - _seen(c, a + i) for a, n in ent for i in range(n))
        rows = sum(a + n - _seen(c, a) for a, n in ent)
        tokens = sum(n for _, n in ent)
        return dict(bytes=rows * c["kv_heads"] * d * 4 + tokens * c["heads"] * d * (6 if c["form"] in ("sigmoid", "blocks") else 4), flops=4 * pairs * c["heads"] * d)
    if c["op"] == "latent":
        ent, W = _entries(c), c["rank"] + c["extra"]
        pairs = sum(a + i + 1 - _seen(c, a + i) for a, n in ent for i in range(n))
        rows, tokens = sum(a + n - _seen(c, a) for a, n in ent), sum(n for _, n in ent)
        return dict(bytes=rows * W * 2 + tokens * c["heads"] * (W + c["rank"]) * 4, flops=2 * pairs * c["heads"] * (W + c["rank"]))
    if c["op"] == "linear":
        n_w = c["n"] * (2 if c["epi"] == "glu" else 1)
        return dict(bytes=2 * c["k"] * (n_w + c["rows"]) + c["rows"] * c["n"] * (4 if c["epi"] == "none" else 2), flops=2 * c["rows"] * c["k"] * n_w)
    if c["op"] == "experts":
        pairs, D, F = c["rows"] * c["top"], c["width"], c["ff"]
        touched = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** c["rows"])
        return dict(bytes=touched * 6 * D * F + c["rows"] * D * 10, flops=6 * pairs * D * F)
    if c["op"] == "recurrence":
        T, H, N, P = c["tokens"], c["heads"], c["n_state"], c["vdim"]
        return dict(bytes=4 * (T * (2 * H * P + 2 * N + H) + c["entries"] * H * N * P), flops=4 * T * H * N * P)
    if c["op"] == "model":
        m, D = MODEL, MODEL["width"]
        lens = _lengths(c["requests"], c["prompt"])
        att, ret = m["heads"] * m["dim"], m["ret_heads"]
        per_layer = D * (2 * att + m["kv_heads"] * m["dim"] + 3 * m["ff"])
        weights = 3 * per_layer + D * ret * (2 * m["ret_dim"] + 3 * m["ret_vdim"])
        head = m["vocab"] * D
        tokens, rows = sum(lens), c["requests"] * (c["steps"] + 1)
        pairs = sum(n * (n + 1) // 2 + c["steps"] * n for n in lens)
        flops = 2 * weights * (tokens + c["requests"] * c["steps"]) + 2 * head * rows + 3 * 4 * pairs * att + 4 * tokens * ret * m["ret_dim"] * m["ret_vdim"]
        return dict(bytes=(1 + c["steps"]) * 2 * (weights + head) + rows * m["vocab"] * 4, flops=flops)
    m = LLAMA
    H = m["heads"] * m["dim"]
    weights, head = m["layers"] * (4 * H * H + 3 * H * m["inter"]), m["vocab"] * H
    tokens, pairs = c["batch"] * (c["prompt"] + c["steps"]), c["batch"] * (c["prompt"] * (c["prompt"] + 1) // 2 + c["steps"] * c["prompt"])
    return dict(bytes=(1 + c["steps"]) * 2 * (weights + head), flops=2 * weights * tokens + 2 * head * c["batch"] * (1 + c["steps"]) + 4 * pairs * H * m["layers"])


def tolerance(c):
    """about four times what two correct results at the same precision differ by (each is off the 64-bit result by the number given)"""
    if c["op"] == "attention":
        return dict(rel=1e-2)      # 2.3e-3: bfloat16 weights and, but for gated heads, bfloat16 outputs
    if c["op"] == "latent":
        return dict(rel=1e-2)      # 1.9e-3: the query and the weights are bfloat16 operands
    if c["op"] == "linear":
        return dict(rel=1e-5) if c["epi"] == "none" else dict(rel=8e-3)   # 4.7e-7 (sums of 32 bits); 1.7e-3 (bfloat16 outputs)
    if c["op"] == "experts":
        return dict(rel=8e-3)      # 1.6e-3: bfloat16 activations between the products
    if c["op"] == "recurrence":
        return dict(rel=1.2e-3)    # 3.1e-4: tf32 operands
    return dict(rel=2.5e-2) if c["op"] == "model" else dict(rel=4e-3)   # 4.3e-3 in bfloat16, 7.2e-4 in fp16


# ---- the same results in 64 bits ---------------------------------------------------------------------------------
def _softmax_rows(s, extra=None):
    """exp(s) / (sum exp(s) + exp(extra)) along the last axis"""
    m = s.amax(-1, keepdim=True)
    if extra is not None:
        m = torch.maximum(m, extra)
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(extra - m) if extra is not None else 0.0))


def _visible(c, a, n, dev="cuda"):
    p, j = torch.arange(a, a + n, device=dev), torch.arange(a + n, device=dev)
    first = torch.tensor([_seen(c, a + i) for i in range(n)], device=dev)
    return (j[None, :] <= p[:, None]) & (j[None, :] >= first[:, None]), p[:, None] - j[None, :]


def _exact_attention(c, seed):
    t, ent, rows, _ = _attention_inputs(c, seed)
    H, G, d, at, out = c["heads"], c["kv_heads"], c["dim"], 0, []
    for b, (a, n) in enumerate(ent):
        q = _f64(t["q"][at:at + n]).reshape(n, H, d)
        k, v = _f64(t["k"][rows[b]]), _f64(t["v"][rows[b]])
        ok, dist = _visible(c, a, n)
        o = torch.empty(n, H, d, dtype=torch.float64, device="cuda")
        for h in range(H):
            g = h // (H // G)
            s = q[:, h] @ k[:, g].T * d ** -0.5
            extra = None
            if c["form"] == "capped":
                s, extra = 50.0 * torch.tanh(s / 50.0), torch.zeros((), dtype=torch.float64, device="cuda")
            elif c["form"] == "biased":
                s, extra = s + _f64(t["bias"][h])[dist.clamp(0, t["bias"].shape[1] - 1)], _f64(t["sink"][h])
            if c["form"] == "sigmoid":
                w = torch.sigmoid(s + _f64(t["head_bias"][h])) * ok
            else:
                w = _softmax_rows(s.masked_fill(~ok, float("-inf")), extra)
            o[:, h] = w @ v[:, g]
        out.append(o.reshape(n, H * d))
        at += n
    return torch.cat(out)


def _exact_latent(c, seed):
    t, ent, rows, _ = _latent_inputs(c, seed)
    at, out = 0, []
    for b, (a, n) in enumerate(ent):
        kv = _f64(t["pool"][rows[b]])
        ok, _ = _visible(c, a, n)
        o = torch.empty(n, c["heads"], c["rank"], dtype=torch.float64, device="cuda")
        for h in range(c["heads"]):
            s = (_f64(t["qa"][at:at + n, h]) @ kv.T * 192 ** -0.5).masked_fill(~ok, float("-inf"))
            o[:, h] = _softmax_rows(s, _f64(t["sink"][h]) if c["sink"] else None) @ kv[:, :c["rank"]]
        out.append(o)
        at += n
    return torch.cat(out)


def _silu(z):
    return z * torch.sigmoid(z)


def _exact_experts(c, seed):
    t = _expert_inputs(c, seed)
    x, h, w = _f64(t["x"]), _f64(t["h"]), _f64(t["weight"])
    for e in range(c["experts"]):
        tok, k = torch.nonzero(t["chosen"] == e, as_tuple=True)
        up = _f64(t["up"][e])
        y = (_silu(h[tok] @ up[:c["ff"]].T) * (h[tok] @ up[c["ff"]:].T)) @ _f64(t["down"][e]).T
        x.index_add_(0, tok, w[tok, k][:, None] * y)
    return x


def _exact_recurrence(c, seed):
    t = _recurrence_inputs(c, seed)
    H, N, P, at, outs, states = c["heads"], c["n_state"], c["vdim"], 0, [], []
    for n in _recurrence_entries(c):
        u = _f64(t["u"][at:at + n])
        x, B, Cc = u[:, :H * P].reshape(n, H, P), u[:, H * P:H * P + N], u[:, H * P + N:]
        dt = torch.nn.functional.softplus(_f64(t["dt"][at:at + n]) + _f64(t["dt_bias"]), threshold=1e9)
        cum = torch.cumsum(dt * _f64(t["A"]), 0)
        cb = Cc @ B.T
        y, st = torch.empty(n, H, P, dtype=torch.float64, device="cuda"), torch.empty(H, N, P, dtype=torch.float64, device="cuda")
        for h in range(H):
            decay = torch.exp((cum[:, None, h] - cum[None, :, h]).tril()).tril()
            y[:, h] = (cb * decay * dt[None, :, h]) @ x[:, h] + _f64(t["D"][h]) * x[:, h]
            st[h] = (B * (torch.exp(cum[-1, h] - cum[:, h]) * dt[:, h])[:, None]).T @ x[:, h]
        outs.append(y.reshape(n, H * P))
        states.append(st)
        at += n
    return [torch.cat(outs), torch.stack(states)]


def _rotate(x, base, interleaved):
    """x [T, heads, d] at positions 0..T-1"""
    T, d = x.shape[0], x.shape[-1]
    f = base ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device="cuda") / d)
    ang = torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * f
    cs, sn = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    u, v = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :d // 2], x[..., d // 2:])
    a, b = u * cs - v * sn, v * cs + u * sn
    return torch.stack([a, b], -1).reshape(x.shape) if interleaved else torch.cat([a, b], -1)


def _rms(x, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps=1e-5):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w + b


def _causal(n):
    return torch.ones(n, n, dtype=torch.bool, device="cuda").tril()


def _exact_model(c, seed):
    m = MODEL
    _, w = _model_weights(seed)
    w = {k: _f64(v) for k, v in w.items()}
    rows = [[] for _ in range(c["steps"] + 1)]
    for seq in _model_tokens(c, seed):
        x, n = w["embed"][torch.tensor(seq, device="cuda").long()], len(seq)
        for i in range(m["layers"]):
            W = {k[len("l%d." % i):]: v for k, v in w.items() if k.startswith("l%d." % i)}
            h = _layer_norm(x, W["norm1"], W["norm1.b"])
            if i < m["layers"] - 1:
                H, G, d = m["heads"], m["kv_heads"], m["dim"]

                def conv(u, taps):
                    pad = torch.cat([torch.zeros(m["taps"] - 1, u.shape[1], dtype=u.dtype, device="cuda"), u])
                    return sum(pad[j:j + n] * taps[:, j] for j in range(m["taps"]))
                q, v = conv(h @ W["mix.q"].T, W["mix.q.conv"]).reshape(n, H, d), conv(h @ W["mix.k"].T, W["mix.k.conv"]).reshape(n, G, d)
                q, k = _rotate(_rms(q) * W["mix.q.norm"], 500000.0, True), _rotate(_rms(v) * W["mix.k.norm"], 500000.0, True)
                k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
                sc = 50.0 * torch.tanh(torch.einsum("thd,nhd->htn", q, k) * d ** -0.5 / 50.0)
                p = _softmax_rows(sc.masked_fill(~_causal(n), float("-inf")), torch.zeros((), dtype=torch.float64, device="cuda"))
                y = torch.einsum("htn,nhd->thd", p, v).reshape(n, H * d) @ W["mix.o"].T
            else:
                H, d, dv = m["ret_heads"], m["ret_dim"], m["ret_vdim"]
                q, k = (_rotate((h @ W["mix." + name].T).reshape(n, H, d), 10000.0, False) for name in ("q", "k"))
                v = (h @ W["mix.v"].T).reshape(n, H, dv)
                decay = torch.tensor([1 - 2.0 ** (-5 - 5 * i / (H - 1)) for i in range(H)], dtype=torch.float32, device="cuda").double()
                back = torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None, :]
                mask = torch.where(back >= 0, decay[:, None, None] ** back.clamp(min=0), 0.0)
                o = torch.einsum("htn,nhv->thv", torch.einsum("thd,nhd->htn", q, k) * d ** -0.5 * mask, v)
                y = (_rms(o).reshape(n, H * dv) * _silu(h @ W["mix.g"].T)) @ W["mix.o"].T
            x = x + 0.5 * _layer_norm(y, W["norm1b"], W["norm1b.b"])
            if i < m["layers"] - 1:
                h = _layer_norm(x, W["norm2"], W["norm2.b"])
                y = (torch.nn.functional.gelu(h @ W["mlp.gate"].T, approximate="tanh") * (h @ W["mlp.up"].T)) @ W["mlp.down"].T
                x = x + 0.5 * _layer_norm(y, W["norm2b"], W["norm2b.b"])
        x = _layer_norm(x[n - c["steps"] - 1:], w["final.norm"], w["final.norm.b"])
        logits = 25.0 * torch.tanh(x @ w["head"].T / 25.0)
        for i in range(c["steps"] + 1):
            rows[i].append(logits[i])
    return [torch.stack(r) for r in rows]


def _exact_llama(c, seed):
    m = LLAMA
    w = {(slot, layer): _f64(t) for slot, layer, t in _llama_weights(seed)}
    H, d = m["heads"], m["dim"]
    rows = [[] for _ in range(c["steps"] + 1)]
    for seq in _llama_tokens(c, seed):
        x, n = w[E.W_EMBED, 0][torch.from_numpy(seq.astype(np.int64)).cuda()], len(seq)
        for i in range(m["layers"]):
            qkv = (_rms(x) * w[E.W_ATTN_NORM, i]) @ w[E.W_QKV, i].T
            q, k, v = qkv.reshape(n, 3, H, d).unbind(1)
            sc = torch.einsum("thd,nhd->htn", _rotate(q, 10000.0, False), _rotate(k, 10000.0, False)) * d ** -0.5
            p = _softmax_rows(sc.masked_fill(~_causal(n), float("-inf")))
            x = x + torch.einsum("htn,nhd->thd", p, v).reshape(n, H * d) @ w[E.W_O, i].T
            gate, up = ((_rms(x) * w[E.W_FFN_NORM, i]) @ w[E.W_GATE_UP, i].T).chunk(2, -1)
            x = x + (_silu(gate) * up) @ w[E.W_DOWN, i].T
        logits = (_rms(x[n - c["steps"] - 1:]) * w[E.W_FINAL_NORM, 0]) @ w[E.W_LM_HEAD, 0].T
        for i in range(c["steps"] + 1):
            rows[i].append(logits[i])
    return [torch.stack(r) for r in rows]


def exact(c, seed):
    if c["op"] == "linear":
        t = _linear_inputs(c, seed)
        y = _f64(t["x"]) @ _f64(t["w"]).T
        return y if c["epi"] == "none" else torch.relu(y) ** 2 if c["epi"] == "relu2" else _silu(y[:, :c["n"]]) * y[:, c["n"]:]
    return dict(attention=_exact_attention, latent=_exact_latent, experts=_exact_experts, recurrence=_exact_recurrence, model=_exact_model,
                llama=_exact_llama)[c["op"]](c, seed)
