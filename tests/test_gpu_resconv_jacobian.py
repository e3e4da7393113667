"""ResConv log-derivatives over lattice sizes, widths and output kinds, against the FP64 oracle's
autograd. Bound: 1e-4 of the sample's largest derivative (FP32 network values and sums; the whole-
network test states 2e-4), and real output with imaginary rows asked for gives zeros there."""
import numpy as np
import pytest
import torch

from oracle import resconv

pytestmark = pytest.mark.gpu


def _pack(s):
    from quantax_gb300.state import pack_spins
    return pack_spins(s)


@pytest.mark.parametrize("C", [4, 8, 12, 16])
@pytest.mark.parametrize("L,B", [(3, 1), (3, 2), (4, 3), (5, 1), (6, 2), (7, 3), (9, 1), (11, 2), (12, 1), (16, 1)])
@pytest.mark.parametrize("out", ["complex", "real", "real_with_im"])
def test_jacobian_shapes(cuda, L, B, C, out):
    from quantax_gb300 import _lib as Lb
    import quantax_gb300 as qtx
    qtx.sites.Square(L)
    cplx, n, ns = out == "complex", L * L, 3
    rng = np.random.default_rng(100 * L + C)
    p = resconv.init_he(B, C, seed=L + C, bias_std=0.1)
    s = (2 * rng.integers(0, 2, (ns, n)) - 1).astype(np.int8)
    pt = torch.as_tensor(p).cuda()
    table = torch.empty(Lb.lib().qgx_resconv_table_floats(B, C), dtype=torch.float32, device="cuda")
    Lb.call("qgx_resconv_prepare", Lb.ptr(pt), B, C, Lb.ptr(table), Lb.stream_ptr())
    ld = p.size + 5  # rows that do not start on 16 bytes
    O = torch.full((2 * ns, ld), float("nan"), dtype=torch.float32, device="cuda")
    ws = torch.empty(Lb.lib().qgx_resconv_jacobian_workspace_bytes(L, B, C), dtype=torch.uint8, device="cuda")
    packed = _pack(s)
    Lb.call("qgx_resconv_jacobian", Lb.ptr(table), L, B, C, int(cplx), Lb.ptr(packed), ns, Lb.ptr(O[:ns]),
            None if out == "real" else Lb.ptr(O[ns:]), ld, Lb.ptr(ws), ws.numel(), Lb.stream_ptr())
    got = O.cpu().numpy().astype(np.float64)
    want = resconv.ResConv(p, L, B, C, cplx).jacobian(s)
    top = np.abs(want).max(axis=1, keepdims=True)
    assert (np.abs(got[:ns, :p.size] - want.real) <= 1e-4 * top).all()
    assert np.isnan(got[:, p.size:]).all()  # nothing written past a row
    if cplx:
        assert (np.abs(got[ns:, :p.size] - want.imag) <= 1e-4 * top).all()
    elif out == "real_with_im":
        assert (got[ns:, :p.size] == 0).all()
    else:
        assert np.isnan(got[ns:]).all()
