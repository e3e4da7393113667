"""Column sums at sizes beside their tiles: the projection A^T y (256-row chunks in four row groups, 256
columns per CTA) and the means of column centring (128-row chunks, 32 columns x 8 chunk groups per
CTA), with rows that start on 16 bytes and rows that do not. Bounds: 2^-44 of the sum of magnitudes for
the float-pair sums (about 48 bits), and two FP32 roundings for the centred entries."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 5), (255, 31), (256, 32), (257, 33), (1025, 255), (130, 257), (2049, 64), (40, 1029)]


def _matrix(rows, cols, pad):
    rng = np.random.default_rng(rows * cols + pad)
    A = rng.standard_normal((rows, cols)).astype(np.float32)
    dev = torch.full((rows, cols + pad), float("nan"), dtype=torch.float32, device="cuda")
    dev[:, :cols] = torch.as_tensor(A).cuda()
    return rng, A.astype(np.float64), dev


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("pad", [0, 3, 4])
def test_projection(cuda, rows, cols, pad):
    from quantax_gb300 import _lib as L
    rng, A, dev = _matrix(rows, cols, pad)
    y = rng.standard_normal(rows)
    yt = torch.as_tensor(y).cuda()
    nb = C.c_int64(0)
    L.call("qgx_obar_rmatvec_workspace_bytes", rows, cols, C.byref(nb))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    x = torch.full((cols + 1,), float("inf"), dtype=torch.float64, device="cuda")
    L.call("qgx_obar_rmatvec", L.ptr(dev), rows, cols, cols + pad, L.ptr(yt), L.ptr(x), L.ptr(ws), ws.numel(),
           L.stream_ptr())
    x = x.cpu().numpy()
    assert np.isposinf(x[cols])
    assert (np.abs(x[:cols] - A.T @ y) <= 2.0 ** -44 * (np.abs(A).T @ np.abs(y))).all()


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("pad", [0, 3])
@pytest.mark.parametrize("weighted", [False, True])
def test_centring(cuda, rows, cols, pad, weighted):
    from quantax_gb300 import _lib as L
    rng, A, dev = _matrix(rows, cols, pad)
    r = rng.uniform(0.5, 1.5, rows) if weighted else np.ones(rows)
    rt = torch.as_tensor(r).cuda() if weighted else None
    ws = torch.empty(L.lib().qgx_center_columns_workspace_bytes(rows, cols), dtype=torch.uint8, device="cuda")
    mean = torch.full((cols + 1,), float("inf"), dtype=torch.float64, device="cuda")
    L.call("qgx_center_columns", L.ptr(dev), rows, cols, cols + pad, L.ptr(rt), L.ptr(mean), L.ptr(ws), ws.numel(),
           L.stream_ptr())
    mean = mean.cpu().numpy()
    assert np.isposinf(mean[cols])
    tol = 2.0 ** -44 * (r @ np.abs(A)) / rows
    assert (np.abs(mean[:cols] - r @ A / rows) <= tol).all()
    f = np.sqrt(r / rows)[:, None]
    want = (A - A.mean(axis=0)) * f
    got = dev[:, :cols].cpu().numpy()
    # the difference, the factor and the product round once each, the difference at the size of its operands
    assert (np.abs(got - want) <= 2.0 ** -22 * f * (np.abs(A) + np.abs(A).mean(axis=0) + 1e-30)).all()
