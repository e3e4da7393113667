"""Tensor-core Grams where the operand rings, the 256-element chunks and the tiles begin, wrap and end.

Bounds, relative to |a_i| |a_j|: the operands' rounding as the Gram tests state it (TF32 2.5e-3,
BF16 1e-2); split TF32 drops lo lo (2^-22) and truncates lo (2 x 2^-22), and one 256-element chunk
accumulated in FP32 by truncation loses at most 256 x 2^-24: 2^-16 together.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOL = {"3xtf32": 2.0 ** -16, "tf32": 2.5e-3, "bf16": 1e-2}


@pytest.mark.parametrize("mode", sorted(TOL))
@pytest.mark.parametrize("rows", [1, 127, 129, 300])
@pytest.mark.parametrize("k", [8, 32, 40, 96, 128, 136, 160, 192, 224, 256, 264, 384, 392, 512, 520, 776, 1032])
def test_gram_ring_edges(cuda, mode, rows, k):
    from quantax_gb300 import _lib as L
    rng = np.random.default_rng(rows * 10007 + k)
    A = rng.normal(size=(rows, k)).astype(np.float32)
    At = torch.as_tensor(A).cuda()
    T = torch.full((rows, rows), np.nan, dtype=torch.float64, device="cuda")
    status = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    if mode == "bf16":
        Ab = torch.empty((rows, k), dtype=torch.bfloat16, device="cuda")
        L.call("qgx_f32_to_bf16", L.ptr(At), rows, k, k, L.ptr(Ab), k, L.stream_ptr())
        L.call("qgx_gram_tc", L.ptr(Ab), 1, rows, k, k, L.ptr(T), rows, L.ptr(status), L.stream_ptr())
    else:
        L.call("qgx_gram_tc", L.ptr(At), 2 if mode == "3xtf32" else 0, rows, k, k, L.ptr(T), rows, L.ptr(status),
               L.stream_ptr())
    got = T.cpu().numpy()
    assert int(status.item()) == 0
    want = A.astype(np.float64) @ A.astype(np.float64).T
    norm = np.linalg.norm(A.astype(np.float64), axis=1)
    assert (np.abs(got - want) <= TOL[mode] * norm[:, None] * norm[None, :]).all()
