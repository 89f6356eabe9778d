"""b200_linear_residual for one row of tiles: 161 to 256 rows against 60 column tiles of 256 or more, ragged in rows, features and K; the rows and widths beside them are refused."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def L(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.capi


def operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, r = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn(M, N, generator=g, device="cuda").half()
    return x, (torch.randn(N, K, generator=g, device="cuda") * K ** -0.5).half(), r


@pytest.mark.parametrize("M,N,K", [(161, 15112, 136), (200, 16000, 264), (256, 15360, 1032)])
@pytest.mark.parametrize("in_place", [False, True])
def test_one_row_of_tiles(L, M, N, K, in_place):
    """the product and the sum are rounded to fp16 (2^-11 each)"""
    x, W, r = operands(M, N, K)
    want, lib = x.double() @ W.double().T + r.double(), L.lib()
    y = r.clone() if in_place else torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    assert lib.b200_linear_residual(x.data_ptr(), W.data_ptr(), (y if in_place else r).data_ptr(), y.data_ptr(), M, N, K, L.F16, None) == 0
    torch.cuda.synchronize()
    assert float((y[:M].double() - want).norm() / want.norm()) < 1e-3
    assert in_place or bool((y[M] == 7.0).all())


@pytest.mark.parametrize("M,N,K", [(160, 15360, 136), (257, 15360, 136), (511, 4096, 136), (200, 15104, 136), (512, 248, 136), (200, 15360, 56)])
def test_what_is_refused(L, M, N, K):
    x, W, r = operands(M, N, K)
    torch.cuda.synchronize()
    assert L.lib().b200_linear_residual(x.data_ptr(), W.data_ptr(), r.data_ptr(), r.data_ptr(), M, N, K, L.F16, None) == -2
