"""The state-space recurrence in chunks of 128 tokens: ends of chunks, of their sixteen-token parts and of column blocks, odd state sizes, groups, carried states,
many turns of the rings, values that are not finite; and the 64-token chunks behind the same call, for leading dimensions that four does not divide and for the workspace
that they need."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
from test_ssd_chunks_gpu import scan  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


class Call:
    def __init__(self, S, H, G, P, N, pad, cnt, seed=0):
        g = torch.Generator(device="cuda").manual_seed(H + N + seed)
        f = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
        self.S, self.H, self.G, self.P, self.N, self.cnt = S, H, G, P, N, cnt
        T, self.ch, E = sum(cnt), H * P + 2 * G * N, len(cnt)
        self.u, self.raw, self.bias, self.A, self.D = f(T, self.ch + pad), f(T, H + 1) * 2 - 2, f(H) * 0.5, -torch.exp(f(H)), f(H)
        self.state = f(E + 1, H, N, P)
        self.before, self.slots, self.start = self.state.double(), list(range(E, 0, -1)), [0 if i % 2 else 7 for i in range(E)]
        self.out = torch.full((T, H * P), float("nan"), device="cuda")
        self.row = [sum(cnt[:i]) for i in range(E)]

    def run(self, room=None):
        S, H, G, P, N, cnt = self.S, self.H, self.G, self.P, self.N, self.cnt
        T, E = sum(cnt), len(cnt)
        ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
        keep = [ints(self.row), ints(list(cnt)), ints(sum([[self.slots[i]] * cnt[i] for i in range(E)], [])), ints(sum([list(range(self.start[i], self.start[i] + cnt[i])) for i in range(E)], []))]
        a = S.SsdScanArgs()
        a.u, a.ld_u, a.x_off, a.b_off, a.c_off = self.u.data_ptr(), self.u.shape[1], 0, H * P, H * P + G * N
        a.dt_raw, a.ld_dt, a.dt_bias, a.A, a.D = self.raw.data_ptr(), H + 1, self.bias.data_ptr(), self.A.data_ptr(), self.D.data_ptr()
        a.state, a.out = self.state.data_ptr(), self.out.data_ptr()
        a.ent_row, a.ent_len, a.slot, a.pos = (k.data_ptr() for k in keep)
        a.n_entries, a.n_tokens, a.heads, a.groups, a.vdim, a.n_state, a.longest_entry, a.chunked = E, T, H, G, P, N, max(cnt), 1
        need = S.lib().b200_ssd_scan_workspace_bytes(T, E, H, G, P, N) if room is None else room
        ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")
        a.workspace, a.workspace_bytes = ws.data_ptr(), need
        torch.cuda.synchronize()
        assert S.lib().b200_ssd_scan(C.byref(a), None) == 0
        torch.cuda.synchronize()

    def check(self):
        v, H, G, P, N = self.u.double(), self.H, self.G, self.P, self.N
        dt = torch.nn.functional.softplus(self.raw[:, :H].double() + self.bias.double(), threshold=1e9)
        for i, n in enumerate(self.cnt):
            r = slice(self.row[i], self.row[i] + n)
            x, B, Cc = v[r, :H * P].reshape(-1, H, P), v[r, H * P:H * P + G * N].reshape(-1, G, N), v[r, H * P + G * N:self.ch].reshape(-1, G, N)
            want, st = scan(x, B, Cc, dt[r], self.A.double(), self.D.double(), self.before[self.slots[i]] if self.start[i] else torch.zeros_like(self.before[0]))
            got = self.out[r].double().reshape(want.shape)
            # tf32 operands: errors of 2^-12 in two factors of every product, about 3e-4 of the result's norm; 1.2e-3 is four times that
            assert float((got - want).norm() / want.norm()) < 1.2e-3, i
            assert float((self.state[self.slots[i]].double() - st).norm() / st.norm()) < 1.2e-3, i
        assert bool((self.state[0].double() == self.before[0]).all())   # the slot nobody used


@pytest.mark.parametrize("H,G,P,N,pad,cnt", [
    (5, 1, 64, 128, 0, (128,)), (6, 2, 64, 33, 2, (129, 127, 1)), (3, 1, 68, 72, 0, (257, 16, 17)), (4, 4, 128, 128, 4, (383, 2)), (2, 1, 4, 100, 0, (640, 130)),
    (64, 1, 64, 128, 0, (300, 200)), (1, 1, 192, 64, 0, (145,))])
def test_chunks_of_128(S, H, G, P, N, pad, cnt):
    """(129, 127, 1) with a leading dimension of 518 falls to the 64-token chunks: test_odd_states has its sizes in chunks of 128"""
    c = Call(S, H, G, P, N, pad, cnt)
    c.run()
    c.check()


def in_chunks_of_128(H, G, P, N, pad, cnt):
    """what ssd_scan_tc asks of a call besides its workspace"""
    return 32 < N <= 128 and P % 4 == 0 and (H * P + 2 * G * N + pad) % 4 == 0 and max(cnt) >= 128


@pytest.mark.parametrize("H,G,P,N,pad,cnt", [(6, 2, 64, 33, 0, (129, 127, 1)), (3, 1, 64, 34, 0, (200, 100)), (5, 1, 68, 127, 2, (256, 131)), (2, 1, 4, 101, 2, (140,)), (4, 4, 64, 67, 0, (385,))])
def test_odd_states(S, H, G, P, N, pad, cnt):
    assert in_chunks_of_128(H, G, P, N, pad, cnt) and N % 4
    c = Call(S, H, G, P, N, pad, cnt)
    c.run()
    c.check()


@pytest.mark.parametrize("H,G,P,N,cnt,most", [(64, 1, 64, 128, (1500, 1300), 11), (33, 1, 64, 128, (2400, 2300), 11), (48, 2, 128, 72, (1100, 1000), 12), (33, 1, 128, 126, (1500, 700, 300, 900), 17),
                                              (72, 1, 72, 64, (520, 1530), 18)])
def test_many_units_per_cta(S, pkg, H, G, P, N, cnt, most):
    """a CTA's rings of sums (four slots), inputs, states and results (two each) go round several times, in some CTAs once more than in others"""
    units = C.CDLL(pkg.lib_path())["_ZN4b20012ssd_tc_unitsEiiiiiii"](sum(cnt), len(cnt), max(cnt), H, G, P, torch.cuda.get_device_properties(0).multi_processor_count)
    per_group = H * ((P + 63) // 64) // G
    blocks = -(-per_group // units)
    assert in_chunks_of_128(H, G, P, N, 0, cnt) and -(-per_group // blocks) == most >= 9
    c = Call(S, H, G, P, N, 0, cnt)
    c.run()
    c.check()


def test_the_smaller_workspace_is_enough(S):
    """a caller that brings what the 64-token chunks need (places of 64 tokens: states, decays, C . B) is served by them"""
    H, P, N, T = 4, 64, 64, 200
    c = Call(S, H, 1, P, N, 0, (T,))
    room = (T // 64 + 2) * (H * N * P + 4 + 64 * 64) * 4 + 256
    assert room < S.lib().b200_ssd_scan_workspace_bytes(T, 1, H, 1, P, N)
    c.run(room)
    c.check()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_are_not_finite_stay_behind_their_token(S, value):
    H, P, N, T, t, h, p = 3, 64, 64, 300, 171, 1, 45
    c = Call(S, H, 1, P, N, 0, (T,))
    clean = Call(S, H, 1, P, N, 0, (T,))
    c.u[t, h * P + p] = value
    c.run()
    clean.run()
    got, want = c.out.reshape(T, H, P), clean.out.reshape(T, H, P)
    hit = torch.zeros_like(got, dtype=torch.bool)
    hit[t:, h, p] = True
    assert bool((got[~hit] == want[~hit]).all()) and not bool(torch.isfinite(got[hit]).any())
    st, ws = c.state[c.slots[0]], clean.state[clean.slots[0]]
    hit = torch.zeros_like(st, dtype=torch.bool)
    hit[h, :, p] = True
    assert bool((st[~hit] == ws[~hit]).all()) and not bool(torch.isfinite(st[hit]).any())
