"""Linears of up to 16 token rows against few weights (fragments straight from global memory): edges of the eight-token tiles, of the 16 features of a CTA, of the
pieces of K, both warp counts, every epilogue."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K,epi,f32", [(8, 8, "none", True), (17, 40, "none", True), (1000, 2048, "relu2", False), (2368, 2056, "none", True), (24, 4104, "none", False),
                                         (128, 264, "glu", True), (384, 2088, "gelu", False), (2048, 1000, "clamp", False), (4096, 2048, "glu", False)])
def test_rows(S, M, N, K, epi, f32):
    """fp32 outputs: chains of at most 128 exact products, every addition of 16 off by at most 2^-23 of the running sum, added up in fp32: below 8 * 2^-23 = 1e-6 of
    the sums' norm, and twice that for the two factors of a gated unit; bfloat16 outputs are rounded by 2^-9 on top"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    gated = epi in ("glu", "gelu", "clamp")
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn((2 if gated else 1) * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    code = dict(none=S.GG_NONE, relu2=S.GG_RELU2, glu=S.GG_GLU, gelu=S.GG_GLU_GELU, clamp=S.GG_GLU_CLAMP)[epi]
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex2(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, code, 0.5 if epi == "clamp" else 0.0, None, 0, None) == 0
    torch.cuda.synchronize()
    z = x.double() @ W.double().T
    if epi == "relu2":
        z = torch.relu(z) ** 2
    elif gated:
        a, b = z[:, :N], z[:, N:]
        if epi == "clamp":
            a, b = a.clamp(max=0.5), b.clamp(-0.5, 0.5)
            z = (b + 1) * a * torch.sigmoid(1.702 * a)
        else:
            z = b * (torch.nn.functional.gelu(a, approximate="tanh") if epi == "gelu" else a * torch.sigmoid(a))
    assert float((y[:M].double() - z).norm() / z.norm()) < (2e-6 if f32 else 4e-3)
    assert bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(6, 1000, 520), (16, 40, 2104)])
def test_rows_fp16_and_bias(pkg, S, M, N, K):
    """fp16 operands and outputs with a bias: outputs rounded by 2^-11"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, b = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(N, generator=g, device="cuda").half()
    W = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).half()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    assert pkg.capi.lib().b200_linear(x.data_ptr(), W.data_ptr(), b.data_ptr(), y.data_ptr(), M, N, K, 1, pkg.capi.F16, None, 0, None) == 0
    torch.cuda.synchronize()
    want = x.double() @ W.double().T + b.double()
    assert float((y[:M].double() - want).norm() / want.norm()) < 1e-3
    assert bool((y[M] == 7.0).all())
