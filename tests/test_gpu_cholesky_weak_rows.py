"""qgx_cholesky on matrices whose rows hardly interact, where it takes its panel in FP64: the entries of
the factor keep FP64's accuracy however small they are.

Bounds. One block (n <= 64), the componentwise bound of an FP64 Cholesky: |L L^T - A|_ij <=
2 (n + 3) 2^-53 (|L| |L|^T)_ij. Past it the tensor-core updates hold a row of a panel to 2^-57 of its
largest entry: with m_i that entry among the panel's columns before column j's block, each panel of K
columns adds at most 4 K 2^-56 m_i m_j. The residual is formed in np.longdouble (64 bits or more)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def factor(A):
    from quantax_gb300 import _lib as L
    n = A.shape[0]
    ws = torch.empty(L.lib().qgx_cholesky_workspace_bytes(n), dtype=torch.uint8, device="cuda")
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    status = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    L.call("qgx_cholesky", L.ptr(A), n, n, L.ptr(info), L.ptr(status), L.ptr(ws), ws.numel(), L.stream_ptr())
    assert int(status.item()) == 0
    return int(info.item())


def check(A):
    n = A.shape[0]
    dev = torch.as_tensor(A).cuda()
    assert factor(dev) == 0
    got = dev.cpu().numpy()
    iu = np.triu_indices(n, 1)
    assert np.array_equal(got[iu], A[iu])
    L = np.tril(got).astype(np.longdouble)
    a = np.abs(L)
    bound = 2 * (n + 3) * np.longdouble(2.0) ** -53 * (a @ a.T)
    for j in range(n):  # column j of the bound: the panels before its block
        for p in range(0, 64 * (j // 64), 256):
            m = a[:, p:min(p + 256, 64 * (j // 64))].max(1)
            bound[:, j] += 4 * 256 * np.longdouble(2.0) ** -56 * m * m[j]
    err = np.abs(L @ L.T - A)
    il = np.tril_indices(n)
    assert (err[il] <= bound[il]).all(), float((err[il] / bound[il]).max())


def coupled(n, c, seed):
    """Diagonal 1 .. 4, couplings c N(0, 1) of sqrt(a_ii a_jj)."""
    r = np.random.default_rng(seed)
    d = r.uniform(1.0, 4.0, n)
    S = np.tril(r.normal(size=(n, n)), -1) * c
    return (S + S.T) * np.sqrt(d[:, None] * d[None, :]) + np.diag(d)


@pytest.mark.parametrize("n", [2, 33, 64, 65, 130, 200])
@pytest.mark.parametrize("c", [1e-4, 1e-6, 1e-12, 1e-150])
def test_weak_couplings(cuda, n, c):
    check(coupled(n, c, n))


@pytest.mark.parametrize("bit", [0, 30, 31, 32, 51, 52])
def test_smallest_couplings(cuda, bit):
    """One bit of the value set: subnormal couplings, and the smallest normal one."""
    n = 70
    c = 2.0 ** (bit - 1074)
    A = torch.full((n, n), c, dtype=torch.float64, device="cuda")
    A.diagonal().fill_(1.0)
    assert factor(A) == 0
    want = torch.full((n, n), c, dtype=torch.float64, device="cuda")
    want.diagonal().fill_(1.0)
    assert torch.equal(A, want)


@pytest.mark.parametrize("scales", [300])
def test_weak_couplings_scaled_rows(cuda, scales):
    A = coupled(130, 1e-6, 7)
    s = np.exp2(np.random.default_rng(8).integers(-scales, scales + 1, 130).astype(float))
    check(A * s[:, None] * s[None, :])  # exact: powers of two


@pytest.mark.parametrize("n,order", [(64, "contiguous"), (64, "interleaved"), (200, "contiguous")])
@pytest.mark.parametrize("c", [1e-6, 1e-12])
def test_groups_that_hardly_interact(cuda, n, order, c):
    r = np.random.default_rng(n)
    G = r.normal(size=(n, n + 8))
    A = G @ G.T / (n + 8) + 1e-3 * np.eye(n)
    group = np.arange(n) * 2 // n if order == "contiguous" else np.arange(n) % 2
    apart = group[:, None] != group[None, :]
    A[apart] *= c
    check(A)


@pytest.mark.parametrize("n", [4500, 7500])
def test_weak_couplings_in_every_launch_form(cuda, n):
    """One and two row tiles per CTA and two launches. |L_ij l_jj - a_ij| <= sum |L_ik| |L_jk| <= 2 n c^2
    and the roundings of one division."""
    c = 1e-12
    g = torch.Generator(device="cuda").manual_seed(n)
    S = (2 * torch.rand((n, n), generator=g, device="cuda", dtype=torch.float64) - 1).tril(-1) * c
    A = S + S.T + torch.eye(n, device="cuda", dtype=torch.float64)
    L = A.clone()
    assert factor(L) == 0
    L = L.tril()
    err = (L.tril(-1) * L.diagonal()[None, :] - A.tril(-1)).abs()
    assert bool((err <= 2 * n * c * c + 4 * 2.0 ** -53 * A.tril(-1).abs()).all())
    assert bool(((L.diagonal() - 1.0).abs() <= 2.0 ** -52).all())


@pytest.mark.parametrize("n", [700, 4500, 7500])
@pytest.mark.parametrize("where", [0.0, 0.0143, 0.5, 0.99, 1.0])
def test_one_weak_row_is_found(cuda, n, where):
    """Couplings of 2^-8 everywhere, of 2^-30 in one row and column: fixed point would keep their
    products to about 2^-61, FP64 to n 2^-83."""
    k = int(where * (n - 1))
    g = torch.Generator(device="cuda").manual_seed(n + k)
    S = (torch.randint(0, 2, (n, n), generator=g, device="cuda", dtype=torch.int8).double() * 2 - 1).tril(-1) * 2.0 ** -8
    A = S + S.T
    w = (1.0 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) * 2.0 ** -30
    A[k], A[:, k] = w, w
    A.diagonal().fill_(1.0)
    L = A.clone()
    assert factor(L) == 0
    L = L.tril()
    err = (L @ L[k] - A[k]).abs()
    err[k] = 0.0
    assert float(err.max()) <= 2.0 ** -66


@pytest.mark.parametrize("n,row", [(64, 40), (300, 200), (300, 5), (7500, 7000)])
def test_minor_that_fails_among_weak_rows(cuda, n, row):
    A = torch.as_tensor(coupled(n, 1e-6, 3) if n < 1000 else np.diag(np.ones(n)) + 1e-6 * (1 - np.eye(n))).cuda()
    A[row, 0] = A[0, row] = 1.5 * float(torch.sqrt(A[0, 0] * A[row, row]))
    assert factor(A) == row + 1
    assert bool(torch.isnan(A.tril()).any())


def test_diagonal_matrix_is_exact(cuda):
    n = 200
    A = torch.diag(torch.exp2(torch.arange(n, device="cuda", dtype=torch.float64) % 7 * 2))
    assert factor(A) == 0
    assert torch.equal(A, torch.diag(torch.exp2(torch.arange(n, device="cuda", dtype=torch.float64) % 7)))
