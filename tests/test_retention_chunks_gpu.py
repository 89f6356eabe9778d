"""The chunk kernels of retention at the sizes that their forms divide: a thread per number up to 32 components, two passes of components above 128, every instance of the
state kernel, exact and ragged, several blocks of value columns, a scan of one number at a time and of four, and of more than eight chunks; carried states."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


def rotate(x, cs, sn, layout):
    """x [T, H, d], the first 2 * cs.shape[1] components rotated"""
    n = cs.shape[1]
    if n == 0:
        return x
    c, s, r = cs[:, None].double(), sn[:, None].double(), x[..., :2 * n]
    u, v = (r[..., :n], r[..., n:]) if layout == "half" else (r[..., 0::2], r[..., 1::2])
    a, b = u * c - v * s, v * c + u * s
    return torch.cat([torch.cat([a, b], -1) if layout == "half" else torch.stack([a, b], -1).flatten(-2), x[..., 2 * n:]], -1)


@pytest.mark.parametrize("heads,dim,vdim,rot_dims,layout,lens", [
    (2, 1, 1, 0, "half", (128, 3)), (3, 4, 8, 4, "half", (130, 64)), (2, 5, 3, 2, "interleaved", (577, 1)), (2, 16, 32, 16, "interleaved", (640,)), (1, 24, 130, 10, "half", (191,)),
    (2, 32, 64, 32, "half", (300, 65)), (1, 33, 35, 32, "interleaved", (200, 129)), (2, 64, 64, 64, "interleaved", (583,)), (1, 100, 96, 64, "half", (150,)),
    (2, 128, 256, 128, "half", (1090, 70)), (1, 127, 129, 126, "interleaved", (140,)), (1, 200, 200, 200, "half", (260,)), (1, 200, 256, 200, "interleaved", (129,)),
    (1, 256, 256, 256, "half", (577, 63)), (1, 256, 260, 130, "interleaved", (135,))])
def test_chunks(S, heads, dim, vdim, rot_dims, layout, lens):
    """fp32 sums of dim products, then of 64 weighted values, then chunk by chunk: (256 + 64 + 18) additions of 2^-24 are 2e-5 at the very most"""
    g = torch.Generator(device="cuda").manual_seed(dim * 1000 + vdim)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    T, E, ld = sum(lens), len(lens), heads * (2 * dim + vdim) + 3
    q_off, k_off, v_off = 1, 1 + heads * dim, 2 + 2 * heads * dim
    proj, ang = f(T, ld), torch.rand(T, rot_dims // 2, generator=g, device="cuda") * 6
    cs, sn = torch.cos(ang).contiguous(), torch.sin(ang).contiguous()
    decay = torch.tensor([0.9, 1.0, 0.995][:heads], device="cuda")
    state, out = f(E + 1, heads, dim, vdim), torch.full((T, heads * vdim), float("nan"), device="cuda")
    before, slots, start, row = state.double(), list(range(E, 0, -1)), [5 if i % 2 == 0 else 0 for i in range(E)], [sum(lens[:i]) for i in range(E)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    keep = [ints(row), ints(list(lens)), ints(sum([[slots[i]] * lens[i] for i in range(E)], [])), ints(sum([list(range(start[i], start[i] + lens[i])) for i in range(E)], []))]
    need = S.lib().b200_retention_workspace_bytes(T, E, heads, dim, vdim)
    ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")
    a = S.RetentionArgs(proj.data_ptr(), ld, q_off, k_off, v_off, cs.data_ptr(), sn.data_ptr(), rot_dims, S.ROPE_HALF if layout == "half" else S.ROPE_INTERLEAVED, decay.data_ptr(),
                        dim ** -0.5, state.data_ptr(), out.data_ptr(), *(k.data_ptr() for k in keep), E, T, heads, dim, vdim, max(lens), ws.data_ptr(), need)
    torch.cuda.synchronize()
    assert need > 0 and max(lens) >= 128 and S.lib().b200_retention(C.byref(a), None) == 0   # (shorter entries are walked token by token)
    torch.cuda.synchronize()
    for i, n in enumerate(lens):
        r = slice(row[i], row[i] + n)
        p = proj[r].double()
        q = rotate(p[:, q_off:q_off + heads * dim].reshape(n, heads, dim), cs[r], sn[r], layout)
        k = rotate(p[:, k_off:k_off + heads * dim].reshape(n, heads, dim), cs[r], sn[r], layout) * dim ** -0.5
        v = p[:, v_off:v_off + heads * vdim].reshape(n, heads, vdim)
        s0 = before[slots[i]] if start[i] else torch.zeros_like(before[0])
        at, d = torch.arange(n, device="cuda"), decay.double()[:, None, None]
        back = at[:, None] - at[None, :]
        w = torch.where(back >= 0, d ** back.clamp(min=0), 0.0) * torch.einsum("thd,nhd->htn", q, k)
        want = torch.einsum("htn,nhv->thv", w, v) + torch.einsum("thd,hdv->thv", q, s0) * (d[:, 0] ** (at + 1.0)).T[:, :, None]
        st = torch.einsum("nhd,nhv->hdv", k * (d[:, 0] ** (n - 1.0 - at)).T[:, :, None], v) + d ** n * s0
        got = out[r].double().reshape(n, heads, vdim)
        assert float((got - want).norm() / want.norm()) < 2e-5, i
        assert float((state[slots[i]].double() - st).norm() / st.norm()) < 2e-5, i
    assert bool((state[0].double() == before[0]).all())   # the slot nobody used
