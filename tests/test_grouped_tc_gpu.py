"""Routed products (b200_gemm_grouped with groups) on the tcgen05 kernel: groups that are empty, that end at, before and behind a block of
rows, feature counts and depths that are no multiple of a tile."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("counts,M", [([1, 0, 2, 5], 8), ([32, 31, 0, 1], 32), ([0, 127, 129, 16, 17, 300], 300), ([0, 0, 0], 40)])
@pytest.mark.parametrize("N,K,epi,f32,gather,scaled", [(256, 128, "none", True, True, False), (200, 72, "none", True, False, True), (64, 200, "glu", False, True, True),
                                                       (192, 1032, "gelu", True, True, False), (130, 64, "relu2", False, True, False)])
def test_groups(S, counts, M, N, K, epi, f32, gather, scaled):
    """fp32 outputs are K exact products added 16 at a time, every addition off by at most 2^-23 of the running sum, 1e-5 for K = 1032 (a
    gated unit multiplies two of them); bfloat16 outputs are rounded by 2^-9"""
    g = torch.Generator(device="cuda").manual_seed(N + K + M)
    T, E, R = 40, len(counts), sum(counts)
    glu = epi in ("glu", "gelu")
    x = torch.randn(max(T, R), K, generator=g, device="cuda").bfloat16()
    W = (torch.randn(E, (2 if glu else 1) * N, K, generator=g, device="cuda") * K ** -0.5).bfloat16()
    off = torch.tensor([sum(counts[:i]) for i in range(E + 1)], dtype=torch.int32, device="cuda")
    src = torch.randint(0, T, (max(R, 1),), generator=g, device="cuda", dtype=torch.int32)
    scale = torch.rand(max(R, 1), generator=g, device="cuda") + 0.5
    y = torch.full((R + 3, N), 7.0, dtype=torch.float32 if f32 else torch.bfloat16, device="cuda")
    a = S.GemmGroupedArgs()
    a.A, a.lda, a.group_off, a.W, a.ldw, a.stride_w = x.data_ptr(), K, off.data_ptr(), W.data_ptr(), K, W.shape[1] * K
    if gather:
        a.a_rows = src.data_ptr()
    if scaled:
        a.row_scale = scale.data_ptr()
    a.C, a.ldc, a.M, a.N, a.K, a.batch, a.trans_b = y.data_ptr(), N, M, N, K, E, 1
    a.epi = dict(none=S.GG_NONE, glu=S.GG_GLU, gelu=S.GG_GLU_GELU, relu2=S.GG_RELU2)[epi]
    a.a_dtype, a.w_dtype, a.c_dtype = S.BF16, S.BF16, S.F32 if f32 else S.BF16
    torch.cuda.synchronize()
    assert S.lib().b200_gemm_grouped(C.byref(a), None) == 0
    torch.cuda.synchronize()
    at = 0
    for e, n in enumerate(counts):
        rows = x[src[at:at + n].long()] if gather else x[at:at + n]
        z = rows.double() @ W[e].double().T * (scale[at:at + n, None].double() if scaled else 1.0)
        if glu:
            act = torch.nn.functional.gelu(z[:, :N], approximate="tanh") if epi == "gelu" else z[:, :N] * torch.sigmoid(z[:, :N])
            z = act * z[:, N:]
        elif epi == "relu2":
            z = torch.relu(z) ** 2
        if n:
            assert float((y[at:at + n].double() - z).norm() / z.norm()) < (2e-5 if f32 else 4e-3), (e, n)
        at += n
    assert bool((y[R:] == 7.0).all())


@pytest.mark.parametrize("N,epi", [(5760, "none"), (2880, "glu"), (7680, "none"), (3840, "glu")])
def test_blocks_of_rows_by_the_number_of_feature_tiles(S, N, epi):
    """270 and 360 feature tiles over all groups: blocks of up to 192 rows, and three CTAs per SM; groups that end at, before and behind such a block. The bounds of test_groups"""
    test_groups(S, [0, 191, 193, 16, 177, 400], 400, N, 136, epi, epi == "none", True, False)
