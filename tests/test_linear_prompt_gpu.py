"""b200_linear_ex with more than 256 token rows (gated units: 128; tokens on the M axis): edges of the row, feature and K tiles, every output and unit."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("M", [257, 512, 513, 1025])
@pytest.mark.parametrize("N,K,epi,f32", [(4096, 2048, "none", True), (1002, 1032, "none", True), (261, 64, "relu2", False), (1000, 136, "none", False),
                                         (256, 2056, "glu", False), (5504, 1024, "glu", True), (1024, 72, "relu2", True)])
def test_many_rows(S, M, N, K, epi, f32):
    """fp32 outputs are K exact products added 16 at a time, every addition off by at most 2^-23 of the running sum (the tensor core
    truncates): K / 16 * 2^-23 = 1.6e-5 for K = 2056; bfloat16 outputs are rounded by 2^-9 on top"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn((2 if epi == "glu" else 1) * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    code = dict(none=S.GG_NONE, relu2=S.GG_RELU2, glu=S.GG_GLU)[epi]
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, code, None, 0, None) == 0
    torch.cuda.synchronize()
    z = x.double() @ W.double().T
    want = z if epi == "none" else torch.relu(z) ** 2 if epi == "relu2" else z[:, :N] * torch.sigmoid(z[:, :N]) * z[:, N:]
    assert float((y[:M].double() - want).norm() / want.norm()) < (1.6e-5 if f32 else 4e-3)
    assert bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M", [129, 159, 257, 300, 1025])
@pytest.mark.parametrize("unit", ["silu", "gelu", "clamp"])
@pytest.mark.parametrize("N,K,f32", [(128, 264, True), (384, 1032, False)])
def test_gated_units_of_ragged_rows(S, M, unit, N, K, f32):
    """Row counts that end inside a warp's 32 rows. The products are off by at most K / 16 * 2^-23 of the sum of their terms' sizes (as above);
    a unit multiplies two of them, silu and gelu move by at most 1.13 of what their argument moves by, 1.702 g by as much again: 8 times
    K / 16 * 2^-23 = 6.2e-5 for K = 1032; bfloat16 outputs are rounded by 2^-9 on top"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(2 * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    code = dict(silu=S.GG_GLU, gelu=S.GG_GLU_GELU, clamp=S.GG_GLU_CLAMP)[unit]
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex2(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, code, 1.5, None, 0, None) == 0
    torch.cuda.synchronize()
    gate, up = (x.double() @ W.double().T).chunk(2, 1)
    if unit == "silu":
        want = gate * torch.sigmoid(gate) * up
    elif unit == "gelu":
        want = torch.nn.functional.gelu(gate, approximate="tanh") * up
    else:
        gate = gate.clamp(max=1.5)
        want = gate * torch.sigmoid(1.702 * gate) * (up.clamp(-1.5, 1.5) + 1)
    assert float((y[:M].double() - want).norm() / want.norm()) < (6.2e-5 if f32 else 4e-3)
    assert bool((y[M] == 7.0).all())
