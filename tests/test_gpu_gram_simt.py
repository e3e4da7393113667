"""FP32 and FP64-sum Gram matrices of vectors in rows (T = A A^T) and in columns (S = A^T A) on the
CUDA cores, at sizes beside the 32, 64 and 128 tiles and the 16-element chunks, with rows that start
on 16 bytes and rows that do not. Bounds: k roundings of 2^-24 per element of |A| |A|^T for FP32
sums, 1e-12 for FP64 ones. The result is exactly symmetric, nothing outside it is written, and a
vector's NaN stays in its row and column."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,pad,off", [(1, 1, 0, 0), (31, 15, 0, 0), (33, 16, 3, 0), (64, 17, 0, 1), (65, 64, 4, 0),
                                         (127, 33, 4, 2), (129, 100, 0, 0), (300, 7, 1, 3), (1056, 203, 1, 0),
                                         (1600, 40, 0, 0), (2050, 29, 3, 1)])
@pytest.mark.parametrize("form", ["rows fp32", "rows fp64", "columns fp32"])
def test_simt_gram(cuda, n, k, pad, off, form):
    from quantax_gb300 import _lib as L
    cols = form.startswith("columns")
    rows, width = (k, n) if cols else (n, k)
    rng = np.random.default_rng(n * k)
    A = rng.standard_normal((rows, width)).astype(np.float32)
    ld = width + pad
    buf = torch.full((rows * ld + off,), float("nan"), dtype=torch.float32, device="cuda")
    dev = buf[off:].view(rows, ld)  # rows start off floats past 16 bytes, NaN between them
    dev[:, :width] = torch.as_tensor(A).cuda()

    def run():
        T = torch.full((n, n + 1), float("inf"), dtype=torch.float64, device="cuda")
        if cols:
            L.call("qgx_gram_t", L.ptr(dev), rows, width, ld, L.ptr(T), n + 1, L.stream_ptr())
        else:
            L.call("qgx_gram", L.ptr(dev), rows, width, ld, L.ptr(T), n + 1,
                   L.GRAM_FP64 if form.endswith("fp64") else L.GRAM_FP32, L.stream_ptr())
        T = T.cpu().numpy()
        assert np.isposinf(T[:, n]).all()
        return T[:, :n]

    V = (A.T if cols else A).astype(np.float64)
    bound = (1e-12 if form.endswith("fp64") else k * 2.0 ** -24) * (np.abs(V) @ np.abs(V).T)
    T = run()
    np.testing.assert_array_equal(T, T.T)
    assert (np.abs(T - V @ V.T) <= bound).all()
    v = n // 2
    if cols:
        dev[0, v] = float("nan")
    else:
        dev[v, 0] = float("nan")
    N = run()
    assert np.isnan(N[v]).all() and np.isnan(N[:, v]).all()
    keep = np.arange(n) != v
    np.testing.assert_array_equal(N[keep][:, keep], T[keep][:, keep])
