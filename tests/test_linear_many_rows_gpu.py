"""Linears of more than 256 token rows: the tiles of one CTA (64, 128, 256 columns) and some of a pair's (test_linear_pair_widths_gpu has them all), ragged in rows, features and K,
plain, squared relu and gated, bfloat16 and fp32 outputs; fp16 with a bias and with a residual."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("M,N,K", [(257, 1000, 1032), (300, 72, 264), (1025, 1032, 520), (1030, 3000, 1032), (2048, 5001, 264), (700, 8200, 136), (385, 24, 72)])
@pytest.mark.parametrize("epi,f32", [("none", True), ("none", False), ("relu2", False), ("relu2", True)])
def test_plain(S, M, N, K, epi, f32):
    """K exact products added 16 at a time, every addition off by at most 2^-23 of the running sum (the tensor core truncates): K / 16 * 2^-23 = 7.7e-6 for K = 1032,
    twice that behind the square; bfloat16 outputs are rounded by 2^-9 on top"""
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


@pytest.mark.parametrize("M,N,K", [(129, 128, 64), (257, 5504, 520), (600, 1024, 2056), (1100, 1408, 264)])
@pytest.mark.parametrize("epi,f32", [("glu", True), ("gelu", False), ("clamp", False), ("glu", False)])
def test_gated(S, M, N, K, epi, f32):
    """as above for two factors; gates of exactly zero, of 90 and of minus 90 (whose exponential overflows) among them"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(2 * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    x[3] = 0
    x[5], W[:8] = 0, 0
    x[5, 0], W[:4, 0], W[4:8, 0] = 9.0, 10.0, -10.0
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    code = dict(glu=S.GG_GLU, gelu=S.GG_GLU_GELU, clamp=S.GG_GLU_CLAMP)[epi]
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex2(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, code, 0.5 if epi == "clamp" else 0.0, None, 0, None) == 0
    torch.cuda.synchronize()
    z = x.double() @ W.double().T
    a, b = z[:, :N], z[:, N:]
    if epi == "clamp":
        a, b = a.clamp(max=0.5), b.clamp(-0.5, 0.5) + 1
        want = b * a * torch.sigmoid(1.702 * a)
    else:
        want = b * (torch.nn.functional.gelu(a, approximate="tanh") if epi == "gelu" else a * torch.sigmoid(a))
    assert float((y[:M].double() - want).norm() / want.norm()) < (3.2e-5 if f32 else 4e-3)
    assert bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(300, 1000, 264), (520, 264, 520), (1100, 4104, 136)])
def test_fp16_bias_and_residual(pkg, S, M, N, K):
    """fp16 outputs: rounded by 2^-11, twice with a residual"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, b, r = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(N, generator=g, device="cuda").half(), torch.randn(M, N, generator=g, device="cuda").half()
    W = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).half()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    z, L = x.double() @ W.double().T, pkg.capi.lib()
    torch.cuda.synchronize()
    assert L.b200_linear(x.data_ptr(), W.data_ptr(), b.data_ptr(), y.data_ptr(), M, N, K, 1, pkg.capi.F16, None, 0, None) == 0
    torch.cuda.synchronize()
    assert float((y[:M].double() - z - b.double()).norm() / z.norm()) < 1e-3
    rc = L.b200_linear_residual(x.data_ptr(), W.data_ptr(), r.data_ptr(), y.data_ptr(), M, N, K, pkg.capi.F16, None)
    torch.cuda.synchronize()
    if M < 512:
        assert rc != 0   # as documented: the caller adds the residual itself
    else:
        assert rc == 0 and float((y[:M].double() - z - r.double()).norm() / z.norm()) < 1.5e-3
    assert bool((y[M] == 7.0).all())
