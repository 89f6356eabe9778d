"""b200_linear_ex with few token rows (the weights stream, a cluster shares a tile's K range): edges of the row, feature and K tiles."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("M", [1, 32, 33, 65, 128, 129, 256])
@pytest.mark.parametrize("N,K,epi,f32", [(4096, 2048, "none", True), (1002, 1032, "none", True), (130, 64, "relu2", False), (40000, 136, "none", False),
                                         (128, 2056, "glu", False), (5504, 1024, "glu", True)])
def test_few_rows(S, M, N, K, epi, f32):
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


@pytest.mark.parametrize("M,N,K,epi,f32", [(33, 30400, 72, "none", True), (64, 30401, 264, "relu2", False), (65, 30404, 1032, "none", False), (128, 30465, 64, "none", True),
                                           (129, 9601, 264, "none", True), (200, 9600, 2056, "relu2", True), (256, 19001, 136, "none", False),
                                           (1, 38000, 64, "none", True), (32, 38017, 1024, "none", False), (32, 38017, 1032, "none", True)])
def test_wide_outputs_of_few_rows(S, M, N, K, epi, f32):
    """more tiles of 128 features than CTAs: each CTA takes several, one after another; ragged rows and features. Tolerances as above"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, S.GG_RELU2 if epi == "relu2" else S.GG_NONE, None, 0, None) == 0
    torch.cuda.synchronize()
    z = x.double() @ W.double().T
    want = torch.relu(z) ** 2 if epi == "relu2" else z
    assert float((y[:M].double() - want).norm() / want.norm()) < (1.6e-5 if f32 else 4e-3)
    assert bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(20, 4100, 520), (100, 30401, 264), (150, 9601, 136)])
def test_bias_and_fp16_outputs(pkg, S, M, N, K):
    """fp16 operands and outputs with a bias, as the LLaMA engine's linears: outputs rounded by 2^-11"""
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
