"""Gated units of every kernel behind b200_linear_ex2 and b200_gemm_grouped: the same bits for few rows (plain division) as for many (a division without a branch)."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


def operands(M, N):
    """x [M, 8] and W [2 N, 8] whose gates are single products of two bfloat16 (exact in fp32) and whose up rows are 1.5: no sum is rounded, whatever its order"""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x, W = torch.zeros(M, 8, device="cuda"), torch.zeros(2 * N, 8, device="cuda")
    x[:, 0] = torch.exp(torch.rand(M, generator=g, device="cuda") * 12 - 8)
    x[: M // 4, 0] = torch.linspace(86.5, 89.5, M // 4, device="cuda")   # denominators from 2^125 to infinity, with the weight -1 below
    x[M // 4, 0], x[M // 4 + 1, 0], x[M // 4 + 2, 0] = 0.0, float("inf"), 1e38
    x[:, 1] = 1.0
    W[:N, 0] = torch.randn(N, generator=g, device="cuda") * 0.5
    W[0, 0], W[1, 0], W[2, 0], W[3, 0] = -1.0, 1.0, -1.0078125, 0.9921875
    W[N:, 1] = 1.5
    return x.bfloat16(), W.bfloat16()


def linear(S, x, W, epi, limit, f32=True):
    M, N = x.shape[0], W.shape[0] // 2
    y = torch.empty(M, N, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    assert S.lib().b200_linear_ex2(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, 8, S.BF16, S.F32 if f32 else S.BF16, epi, limit, None, 0, None) == 0
    torch.cuda.synchronize()
    return y


def few_rows(S, x, W, epi, limit, f32=True):
    return torch.cat([linear(S, x[i:i + 8].contiguous(), W, epi, limit, f32) for i in range(0, x.shape[0], 8)])


def same(a, b):
    return bool(((a == b) | (a.isnan() & b.isnan())).all())


# one CTA of 256 columns, pairs of 128 to 256 columns (what choose_tile names for 8 products: the narrowest that fills the chip), the weight-streaming kernel
@pytest.mark.parametrize("M,N", [(257, 128), (600, 1024), (2048, 5504), (4100, 384), (100, 256)])
@pytest.mark.parametrize("unit", ["silu", "clamp"])
def test_the_same_bits_for_few_and_many_rows(S, M, N, unit):
    x, W = operands(M, N)
    epi, limit = (S.GG_GLU, 0.0) if unit == "silu" else (S.GG_GLU_CLAMP, 100.0)
    got = linear(S, x, W, epi, limit)
    assert same(got, few_rows(S, x, W, epi, limit))
    if unit == "silu":   # gates of which a division by more than 2^126 would make zero
        z = x[:, :1].double() @ W[:N, :1].double().T
        want = 1.5 * z / (1 + torch.exp(-z))
        at = (z > -88.7) & (z < -80)
        assert int(at.sum()) > 0
        # expf is off by 2^-23, the sum, the quotient and the product by 2^-24 each: less than 2^-21 in all
        assert float(((got.double() - want).abs() / want.abs())[at].max()) < 2.0 ** -21


@pytest.mark.parametrize("rows", [7, 40, 300])
@pytest.mark.parametrize("unit", ["silu", "clamp"])
def test_the_same_bits_for_routed_rows(S, rows, unit):
    N = 192
    x, W = operands(rows, N)
    epi, limit = (S.GG_GLU, 0.0) if unit == "silu" else (S.GG_GLU_CLAMP, 100.0)
    off = torch.tensor([0, rows], dtype=torch.int32, device="cuda")
    y = torch.empty(rows, N, device="cuda")
    a = S.GemmGroupedArgs()
    a.A, a.lda, a.group_off, a.W, a.ldw, a.stride_w = x.data_ptr(), 8, off.data_ptr(), W.data_ptr(), 8, 2 * N * 8
    a.C, a.ldc, a.M, a.N, a.K, a.batch, a.trans_b, a.epi, a.epi_param = y.data_ptr(), N, rows, N, 8, 1, 1, epi, limit
    a.a_dtype = a.w_dtype = S.BF16
    a.c_dtype = S.F32
    torch.cuda.synchronize()
    assert S.lib().b200_gemm_grouped(C.byref(a), None) == 0
    torch.cuda.synchronize()
    assert same(y, few_rows(S, x, W, epi, limit))


def test_gelu_is_no_further_off_than_by_tanh(S):
    """few rows take tanhf; the tiles' form has to be as near to 64 bits, in the norm and (a sixteenth of slack) at the worst gate that is not tiny"""
    M, N = 600, 1024
    x, W = operands(M, N)
    x[M // 4 + 1:M // 4 + 3] = 0
    z = x[:, :1].double() @ W[:N, :1].double().T
    want = 1.5 * torch.nn.functional.gelu(z, approximate="tanh")
    tiles, few = linear(S, x, W, S.GG_GLU_GELU, 0.0).double(), few_rows(S, x, W, S.GG_GLU_GELU, 0.0).double()
    assert float((tiles - want).norm()) <= float((few - want).norm())
    at = (z.abs() < 4) & (z.abs() > 1e-3)
    assert float(((tiles - want).abs() / want.abs())[at].max()) <= 1.0625 * float(((few - want).abs() / want.abs())[at].max())


@pytest.mark.parametrize("M,N", [(257, 128), (600, 1024), (1100, 5504)])
def test_fp16_gives_the_bits_of_the_unfused_sequence(pkg, S, M, N):
    """the product rounded to fp16, silu of the gate rounded, their product rounded; sums are single products"""
    x, W = (t.clamp(-90, 90).half() for t in operands(M, N))
    x[M // 4 + 1] = 0
    y, capi = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda"), pkg.capi
    torch.cuda.synchronize()
    assert capi.lib().b200_linear_swiglu(x.data_ptr(), W.data_ptr(), y.data_ptr(), M, N, 8, capi.F16, None) == 0
    torch.cuda.synchronize()
    z = (x.float() @ W.float().T).half().float()
    g, u = z[:, :N], z[:, N:]
    assert same(y[:M], ((g / (1 + torch.exp(-g))).half().float() * u).half())
    assert bool((y[M] == 7.0).all())
