"""The state-space recurrence on numbers near the end of fp32's range: products, states and C . B of more than 2^114, finite in the result."""
import pytest

torch = pytest.importorskip("torch")
from test_ssd_tc_gpu import Call  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S(pkg):
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return pkg.serve


@pytest.mark.parametrize("x,b,c", [(2e35, 1e-10, 1e10), (1e16, 1e20, 1e-20), (1e-20, 1e18, 1e18)])
@pytest.mark.parametrize("H,P,N,cnt", [(3, 64, 128, (300, 260)), (2, 68, 40, (150,))])
def test_large_numbers_stay_finite(S, H, P, N, cnt, x, b, c):
    """large steps times inputs; large states; large C . B: a power of ten on one operand and its inverse on another leave the relative error as it is (1.2e-3: test_ssd_tc_gpu)"""
    call = Call(S, H, 1, P, N, 0, cnt)
    call.u[:, :H * P] *= x
    call.u[:, H * P:H * P + N] *= b
    call.u[:, H * P + N:] *= c
    call.state *= x * b
    call.before = call.state.double()
    largest = max(float(call.u[:, :H * P].abs().max()) * 0.05, float(call.before.abs().max()), b * c)
    assert largest > 2.0 ** 114   # what this test is about
    call.run()
    assert bool(torch.isfinite(call.out).all())
    call.check()
