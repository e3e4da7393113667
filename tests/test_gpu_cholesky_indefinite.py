"""qgx_cholesky on matrices that one entry makes indefinite: whatever the ratio of that entry to
sqrt(a_ii a_jj), info is the order of the first leading minor that fails and the factor holds NaN from
there (an entry whose scaled value exceeds 1 must not pass for a small one)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def factor(A):
    from quantax_gb300 import _lib as L
    n = A.shape[0]
    ws = torch.empty(L.lib().qgx_cholesky_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    L.call("qgx_cholesky", L.ptr(A), n, n, L.ptr(info), None, L.ptr(ws), ws.numel(), L.stream_ptr())
    return int(info.item())


# within 32 rows, across the halves of a block, in its lower half, below it, in a later panel; n = 7500
# also takes the first blocks' two-launch form
@pytest.mark.parametrize("n,row,col", [(64, 9, 4), (64, 50, 7), (64, 60, 40), (300, 130, 20), (600, 400, 300),
                                       (7500, 20, 3), (7500, 7300, 30)])
@pytest.mark.parametrize("scale", [-37, 0, 1, 200])
def test_indefinite_two_by_two_minor(cuda, n, row, col, scale):
    A = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    d = torch.ones(n, dtype=torch.float64, device="cuda")
    d[row] = 1.96
    ratios = [1.0001, 1.5, 1.9, 2.0, 2.8 / 1.4, 2.9 / 1.4, 2.3, 2.6, 2.9, 3.5] if n < 7500 else [2.8 / 1.4, 2.5]
    for r in ratios:
        for sign in (1.0, -1.0):
            A.zero_()
            A.diagonal().copy_(d * 2.0 ** scale)
            A[row, col] = A[col, row] = sign * r * 1.4 * 2.0 ** scale
            assert factor(A) == row + 1, (r, sign)
            assert bool(torch.isnan(A[row, :row + 1]).any())
    A.zero_()  # the definite neighbour
    A.diagonal().copy_(d * 2.0 ** scale)
    A[row, col] = A[col, row] = 0.999 * 1.4 * 2.0 ** scale
    assert factor(A) == 0
    assert abs(float(A[row, col]) / 2.0 ** (scale / 2) - 0.999 * 1.4) <= 2.0 ** -50
    assert not bool(torch.isnan(A).any())
