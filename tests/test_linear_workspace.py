"""The linears need no scratch: their size functions say 0, so that no caller allocates (or waits, or drops a captured step) for it."""
import pytest


@pytest.mark.parametrize("rows,n,k", [(1, 4096, 2048), (8, 4096, 2048), (200, 2048, 8192), (256, 32000, 4096), (300, 4096, 2048)])
def test_linears_ask_for_no_workspace(pkg, rows, n, k):
    assert pkg.serve.lib().b200_linear_ex_workspace_bytes(rows, n, k) == 0
    assert pkg.capi.lib().b200_linear_workspace_bytes(rows, n, k, 1, pkg.capi.F16) == 0
