"""The chunk form of the state-space recurrence: entries around the ends of chunks and of their sixteen-row parts, carried states, groups, odd leading dimensions."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


def scan(x, B, Cc, dt, A, D, st):
    """token by token in 64 bits: x [n, H, P], B and Cc [n, G, N], dt [n, H], st [H, N, P]"""
    r, out = x.shape[1] // B.shape[1], []
    for i in range(len(x)):
        b, c = B[i].repeat_interleave(r, 0), Cc[i].repeat_interleave(r, 0)
        st = torch.exp(A * dt[i])[:, None, None] * st + (dt[i][:, None] * b)[:, :, None] * x[i][:, None, :]
        out.append((c[:, :, None] * st).sum(1) + D[:, None] * x[i])
    return torch.stack(out), st


@pytest.mark.parametrize("H,G,P,N,pad,cnt", [(48, 1, 64, 128, 0, (150, 128)), (48, 2, 64, 64, 4, (129, 63, 150)), (24, 3, 128, 128, 8, (65, 191, 1, 80)), (40, 1, 64, 128, 0, (1025,)), (16384, 16384, 1, 4, 0, (130,))])
def test_chunk_borders(S, H, G, P, N, pad, cnt):
    """The last case has more groups than a quarter of what a grid's y or z can count. tf32 operands: errors of 2^-12 in two factors of every product, about 3e-4 of the result's norm; 1.2e-3 is four times that"""
    g = torch.Generator(device="cuda").manual_seed(H + N)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    T, ch, E = sum(cnt), H * P + 2 * G * N, len(cnt)
    u, raw, bias, A, D = f(T, ch + pad), f(T, H + 1) * 2 - 2, f(H) * 0.5, -torch.exp(f(H)), f(H)
    state = f(E + 1, H, N, P)
    before, slots, start = state.double(), list(range(E, 0, -1)), [0 if i % 2 else 7 for i in range(E)]
    out = torch.full((T, H * P), float("nan"), device="cuda")
    row = [sum(cnt[:i]) for i in range(E)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    keep = [ints(row), ints(list(cnt)), ints(sum([[slots[i]] * cnt[i] for i in range(E)], [])), ints(sum([list(range(start[i], start[i] + cnt[i])) for i in range(E)], []))]
    a = S.SsdScanArgs()
    a.u, a.ld_u, a.x_off, a.b_off, a.c_off = u.data_ptr(), ch + pad, 0, H * P, H * P + G * N
    a.dt_raw, a.ld_dt, a.dt_bias, a.A, a.D = raw.data_ptr(), H + 1, bias.data_ptr(), A.data_ptr(), D.data_ptr()
    a.state, a.out = state.data_ptr(), out.data_ptr()
    a.ent_row, a.ent_len, a.slot, a.pos = (k.data_ptr() for k in keep)
    a.n_entries, a.n_tokens, a.heads, a.groups, a.vdim, a.n_state, a.longest_entry, a.chunked = E, T, H, G, P, N, max(cnt), 1
    need = S.lib().b200_ssd_scan_workspace_bytes(T, E, H, G, P, N)
    ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    torch.cuda.synchronize()
    assert S.lib().b200_ssd_scan(C.byref(a), None) == 0
    torch.cuda.synchronize()
    v = u.double()
    dt = torch.nn.functional.softplus(raw[:, :H].double() + bias.double(), threshold=1e9)
    for i in range(E):
        r = slice(row[i], row[i] + cnt[i])
        x, B, Cc = v[r, :H * P].reshape(-1, H, P), v[r, H * P:H * P + G * N].reshape(-1, G, N), v[r, H * P + G * N:ch].reshape(-1, G, N)
        want, st = scan(x, B, Cc, dt[r], A.double(), D.double(), before[slots[i]] if start[i] else torch.zeros_like(before[0]))
        got = out[r].double().reshape(want.shape)
        assert float((got - want).norm() / want.norm()) < 1.2e-3, i
        assert float((state[slots[i]].double() - st).norm() / st.norm()) < 1.2e-3, i
    assert bool((state[0].double() == before[0]).all())   # the slot nobody used
