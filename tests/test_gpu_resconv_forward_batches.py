"""FP32 ResConv forward over batch lengths and table alignments. A configuration's log psi does not
depend on the batch that holds it (one CTA per few configurations, more CTAs than fit on the chip,
a ragged last one), nor on whether the table starts on 16 bytes (the layers' weights are staged 16
bytes at a time where it does): the same bits. Rows against the FP64 oracle within 1e-4, the bound
of the network's other FP32 tests."""
import numpy as np
import pytest
import torch

from oracle import resconv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,B,C,cplx,ns", [(10, 2, 16, True, 5 * 608 + 3), (4, 2, 8, True, 20011), (7, 2, 16, True, 4001),
                                           (6, 3, 12, False, 5003), (12, 1, 4, True, 1501), (16, 1, 16, True, 911),
                                           (3, 1, 4, False, 1), (4, 1, 12, True, 2)])
def test_forward_batches(cuda, L, B, C, cplx, ns):
    from quantax_gb300 import _lib as Lb
    from quantax_gb300.state import pack_spins
    import quantax_gb300 as qtx
    qtx.sites.Square(L)
    p = resconv.init_he(B, C, seed=L + C, bias_std=0.1)
    rng = np.random.default_rng(ns)
    s = (2 * rng.integers(0, 2, (ns, L * L)) - 1).astype(np.int8)
    pt = torch.as_tensor(p).cuda()
    nt = Lb.lib().qgx_resconv_table_floats(B, C)
    table = torch.empty(nt, dtype=torch.float32, device="cuda")
    Lb.call("qgx_resconv_prepare", Lb.ptr(pt), B, C, Lb.ptr(table), Lb.stream_ptr())

    def run(tab, rows):
        packed = pack_spins(rows)
        out = torch.full((len(rows), 2), float("nan"), dtype=torch.float32, device="cuda")
        Lb.call("qgx_resconv_log_psi", Lb.ptr(tab), L, B, C, int(cplx), 0, Lb.ptr(packed), len(rows), Lb.ptr(out),
                Lb.stream_ptr())
        return out.cpu().numpy()

    whole = run(table, s)
    for cut in (1, 2, 7):
        np.testing.assert_array_equal(run(table, s[:cut]), whole[:cut])
        np.testing.assert_array_equal(run(table, s[-cut:]), whole[-cut:])
    shifted = torch.empty(nt + 1, dtype=torch.float32, device="cuda")[1:]
    shifted.copy_(table)
    np.testing.assert_array_equal(run(shifted, s), whole)
    rows = np.unique(np.linspace(0, ns - 1, 9).astype(int))
    want = resconv.ResConv(p, L, B, C, cplx).log_psi(s[rows])
    got = whole[rows, 0].astype(np.float64) + 1j * whole[rows, 1]
    assert np.abs(got.real - want.real).max() < 1e-4
    assert np.abs(np.angle(np.exp(1j * (got.imag - want.imag)))).max() < 1e-4
