"""The combination of routed experts: a block of as many threads as a row has pieces of four columns, one and several blocks per row, one to eight experts, experts without a
row, and what falls to the kernel that goes column by column (nine experts, widths that four does not divide, rows that do not lie on 16 bytes)."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("T,width", [(3, 4), (40, 24), (9, 128), (5, 132), (300, 1024), (7, 1028), (33, 2052), (4, 26)])
@pytest.mark.parametrize("top", [1, 3, 4, 5, 7, 8, 9])
@pytest.mark.parametrize("f32,extras,shift", [(False, False, 0), (True, True, 0), (False, True, 1)])
def test_combine(S, T, width, top, f32, extras, shift):
    g = torch.Generator(device="cuda").manual_seed(T * width + top)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    room = f(T * width + shift)
    x = room[shift:].reshape(T, width)
    mix, shared = (f(T, width), f(T, width)) if extras else (None, None)
    eo, h = f(T * top, width), f(T, width).to(torch.float32 if f32 else torch.bfloat16)
    dest = torch.randperm(T * top, generator=g, device="cuda").to(torch.int32).reshape(T, top)
    dest = torch.where(torch.rand(T, top, generator=g, device="cuda") < 0.2, -1, dest).to(torch.int32).contiguous()
    w = torch.rand(T, top, generator=g, device="cuda")
    rows = torch.where((dest >= 0)[:, :, None], eo[dest.clamp(min=0).long()], h.float()[:, None, :]).double()
    parts = [x.double()] + ([mix.double(), shared.double()] if extras else []) + [(w.double()[:, :, None] * rows).sum(1)]
    want, size = sum(parts), sum(p.abs() for p in parts[:-1]) + (w.double()[:, :, None] * rows.abs()).sum(1)
    torch.cuda.synchronize()
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    assert S.lib().b200_residual_combine(p(x), p(mix), p(shared), p(eo), p(dest), p(w), p(h), S.F32 if f32 else S.BF16, T, width, top, None) == 0
    torch.cuda.synchronize()
    # top + 3 additions in fp32, each off by 2^-24 of what has been added up
    assert bool(((x.double() - want).abs() <= (top + 3) * 2.0 ** -24 * size).all())
