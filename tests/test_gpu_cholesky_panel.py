"""The fixed-point panel of the FP64 Cholesky (qgx_cholesky): block edges, row scales, matrices
that are not positive definite and entries that are not numbers.

Bound of the factor: |L L^T - A|_ij <= 8 (n + 1) 2^-53 sqrt(a_ii a_jj), eight times the standard
bound of an FP64 Cholesky (the residual is evaluated in FP64 itself).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def factor(A):
    from quantax_gb300 import _lib as L
    n = A.shape[0]
    At = torch.as_tensor(np.ascontiguousarray(A)).cuda()
    ws = torch.empty(max(L.lib().qgx_cholesky_workspace_bytes(n), 256), dtype=torch.uint8, device="cuda")
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    L.call("qgx_cholesky", L.ptr(At), n, n, L.ptr(info), None, L.ptr(ws), ws.numel(), L.stream_ptr())
    return At.cpu().numpy(), int(info.item())


def spd(n, seed, k=None):
    rng = np.random.default_rng(seed)
    G = rng.normal(size=(n, k or n + 8))
    return G @ G.T / G.shape[1] + 1e-3 * np.eye(n)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 127, 129, 192, 255, 256, 257, 319, 321, 513, 545])
@pytest.mark.parametrize("scales", [0, 300])
def test_block_edges_and_row_scales(cuda, n, scales):
    A = spd(n, n)
    s = np.exp2(np.random.default_rng(n + 1).integers(-scales, scales + 1, n).astype(float))
    A = A * s[:, None] * s[None, :]  # exact: powers of two
    Lf, info = factor(A)
    assert info == 0
    L = np.tril(Lf) / s[:, None]  # back to the unscaled matrix, exactly
    B = A / s[:, None] / s[None, :]
    d = np.sqrt(np.diag(B))
    assert (np.abs(L @ L.T - B) <= 8 * (n + 1) * 2.0 ** -53 * d[:, None] * d[None, :]).all()
    iu = np.triu_indices(n, 1)
    assert np.array_equal(Lf[iu], A[iu])


@pytest.mark.parametrize("row,col", [(1, 0), (40, 3), (63, 62), (64, 0), (200, 100), (300, 299), (511, 5)])
@pytest.mark.parametrize("excess", [1.0001, 3.0, 1e6, 1e200])
def test_row_beyond_its_bound_is_reported(cuda, row, col, excess):
    """|a_ij| > sqrt(a_ii a_jj): the first leading minor that fails is row + 1's, whether row i
    leaves the range of the fixed-point entries or only turns its pivot negative."""
    n = 512
    A = np.diag(np.full(n, 2.0))
    A[row, col] = A[col, row] = 2.0 * excess
    Lf, info = factor(A)
    assert info == row + 1
    assert np.isnan(np.tril(Lf)).any()  # what is solved with it is not a number


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 0.0, -1.0])
@pytest.mark.parametrize("row", [0, 63, 64, 400])
def test_bad_diagonal_entry(cuda, row, bad):
    n = 448
    A = spd(n, 3)
    A[row, row] = bad
    Lf, info = factor(A)
    assert info == row + 1
    assert np.isnan(np.tril(Lf)).any()


@pytest.mark.parametrize("row,col", [(10, 2), (100, 2), (400, 300)])
def test_nan_entry_reaches_the_factor(cuda, row, col):
    A = spd(448, 4)
    A[row, col] = A[col, row] = np.nan
    Lf, _ = factor(A)
    assert np.isnan(Lf[row, :row + 1]).any()


def test_leading_blocks_do_not_depend_on_the_rows_below(cuda):
    """The rows below a diagonal block decide how its factorisation and the triangular solve are
    launched (together with one or two row tiles per CTA, or one after the other). The factor of a
    leading submatrix is the leading part of the whole factor, bit for bit, whichever it was."""
    n = 7700
    g = torch.Generator(device="cuda").manual_seed(5)
    G = torch.randn((n, 300), generator=g, device="cuda", dtype=torch.float64)
    A = (G @ G.T / 300 + torch.eye(n, device="cuda", dtype=torch.float64)).cpu().numpy()
    whole, info = factor(A)
    assert info == 0
    for m in (7297, 5000, 2500, 2496, 2433, 700):
        part, info = factor(A[:m, :m])
        assert info == 0
        assert np.array_equal(np.tril(part), np.tril(whole[:m, :m]))
