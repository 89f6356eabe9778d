"""Linears of many token rows on pairs of CTAs whose tiles are 128, 160, 192, 224 or 256 columns wide: shapes for which the rule names each width, ragged in rows, features
and K, so that a tile ends inside a group of columns, behind the last feature (gated: where the rows of the next half begin) and behind the last token."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


def _run(S, M, N, K, epi, f32, n_w):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(n_w, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, S.BF16, S.F32 if f32 else S.BF16, epi, None, 0, None) == 0
    torch.cuda.synchronize()
    assert bool((y[M] == 7.0).all())
    return x.double() @ W.double().T, y[:M].double()


# every addition of 16 products off by at most 2^-23 of the running sum: K / 16 * 2^-23 = 1.6e-5 for K = 2056; bfloat16 outputs rounded by 2^-9 on top, gated ones are
# two such factors
@pytest.mark.parametrize("M,N,K,f32", [(1073, 5600, 1032, False), (425, 4752, 1032, False), (264, 6944, 1032, False), (520, 4800, 2056, False), (1077, 7068, 2056, False),
                                       (1079, 7096, 520, True), (533, 3785, 520, True), (260, 6488, 1032, True), (274, 7145, 2056, True), (1050, 7076, 2056, True)])
def test_plain(S, M, N, K, f32):
    want, got = _run(S, M, N, K, S.GG_NONE, f32, N)
    assert float((got - want).norm() / want.norm()) < (1.6e-5 if f32 else 4e-3)


@pytest.mark.parametrize("M,N,K,f32", [(324, 128, 520, False), (285, 2432, 1032, False), (263, 3072, 1032, False), (264, 3840, 2056, False), (795, 4224, 2056, False),
                                       (266, 128, 520, True), (266, 2560, 1032, True), (269, 3072, 1032, True), (267, 3712, 2056, True), (150, 5504, 1032, False)])
def test_gated(S, M, N, K, f32):
    z, got = _run(S, M, N, K, S.GG_GLU, f32, 2 * N)
    want = z[:, N:] * z[:, :N] * torch.sigmoid(z[:, :N])
    assert float((got - want).norm() / want.norm()) < (3.2e-5 if f32 else 4e-3)


@pytest.mark.parametrize("M,N,K", [(520, 11008, 264), (300, 3712, 2056), (700, 4096, 136)])
def test_fp16_gated(pkg, S, M, N, K):
    """the same rounding points as the product followed by the gated unit, each 2^-11"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").half()
    W = (torch.randn(2 * N, K, generator=g, device="cuda") * K ** -0.5).half()
    y = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    assert pkg.capi.lib().b200_linear_swiglu(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, K, pkg.capi.F16, None) == 0
    torch.cuda.synchronize()
    z = x.double() @ W.double().T
    want = z[:, N:] * z[:, :N] * torch.sigmoid(z[:, :N])
    assert float((y[:M].double() - want).norm() / want.norm()) < 2e-3
    assert bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(513, 4096, 1032), (700, 2048, 4104), (1522, 2056, 1032), (520, 520, 264)])
def test_fp16_residual_in_place(pkg, S, M, N, K):
    """the residual is read ahead of the sums it is added to, and the outputs may take its place"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, K, generator=g, device="cuda").half()
    W = (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).half()
    r = torch.randn(M, N, generator=g, device="cuda").half()
    y = r.clone()
    torch.cuda.synchronize()
    assert pkg.capi.lib().b200_linear_residual(x.data_ptr(), W.data_ptr(), y.data_ptr(), y.data_ptr(), M, N, K, pkg.capi.F16, None) == 0
    torch.cuda.synchronize()
    want = x.double() @ W.double().T + r.double()
    assert float((y.double() - want).norm() / want.norm()) < 1.5e-3
