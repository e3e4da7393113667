"""Local energies of a ResConv whose amplitude ratios overflow: the imaginary part of an overflowing
ratio times a phase of zero is not a number, as the complex product has it, and stays zero elsewhere."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import metropolis
from test_gpu_resconv import Net, _pack

pytestmark = pytest.mark.gpu


def test_overflowing_ratios_of_a_real_network(cuda):
    import quantax_gb300.operator as O
    from quantax_gb300 import _lib as Lb
    L, B, Cc, ns = 4, 2, 8, 40
    n = L * L
    net = Net(L, B, Cc, False, seed=5)
    net.pt[-9 * Cc * Cc:] *= 1500.0  # the last layer: log ratios up to 1150
    Lb.call("qgx_resconv_prepare", Lb.ptr(net.pt), B, Cc, Lb.ptr(net.table), Lb.stream_ptr())
    op = O.CompiledOperator(*O.compile_op_list([["x", [[1.0, i] for i in range(n)]]]))
    s = metropolis.init_uniform(ns, n, 9)
    flips = np.repeat(s[:, None], n, 1)
    flips[:, np.arange(n), np.arange(n)] *= -1
    here, there = net.log_psi(_pack(s)), net.log_psi(_pack(flips.reshape(-1, n))).reshape(ns, n)
    assert (here.imag == 0).all() and (there.imag == 0).all()
    over = ((there.real - here.real[:, None]) > 710).any(1)
    clear = ((there.real - here.real[:, None]) < 709).all(1)
    assert over.any() and clear.any()
    ws = torch.empty(Lb.lib().qgx_resconv_eloc_workspace_bytes(L, ns, n), dtype=torch.uint8, device="cuda")
    er, ei = (torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(2))
    Lb.call("qgx_resconv_eloc", Lb.ptr(net.table), L, B, Cc, 0, 0, C.byref(op.struct), Lb.ptr(_pack(s)), ns,
            Lb.ptr(er), Lb.ptr(ei), Lb.ptr(ws), ws.numel(), Lb.stream_ptr())
    er, ei = er.cpu().numpy(), ei.cpu().numpy()
    assert np.isinf(er[over]).all() and np.isnan(ei[over]).all()
    assert np.isfinite(er[clear]).all() and (ei[clear] == 0).all()
