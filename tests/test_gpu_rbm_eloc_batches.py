"""RBM local energies over site counts, hidden widths and batch lengths. One warp takes one sample or
two (long batches, up to 512 hidden units), four flips at a time and 32 operator terms per pass:
counts beside each of those, terms whose element is zero for one spin direction, and operators with
every kind of term. A sample's value does not depend on its batch (the same bits), and rows agree
with the FP64 oracle within 2e-5 of the largest: a log ratio sums FP32 rounding of at most m = 2000
terms whose slopes are below 0.2."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import lattice, metropolis, operators as oops, rbm
from test_gpu_rbm import Rbm, compiled, lib, pack

pytestmark = pytest.mark.gpu


def _ops(kind, N):
    bonds = lattice.neighbors((N,), 1)
    if kind == "flips":  # fields on all sites, and couplings
        return oops.chain_tfim(N, h=0.7, J=1.2)
    if kind == "bonds":  # exchange and z z on all bonds
        return oops.heisenberg_op_list([bonds], [1.0], [1], False)
    sites = range(0, N, 3)
    return [["x", [[0.4 + 0.1 * i, i] for i in sites]], ["z", [[0.3, i] for i in range(N)]],
            ["+", [[0.2, i] for i in sites]], ["xx", [[0.25, 0, N - 1]]], ["zz", [[-0.5, 0, N - 1]]]]


@pytest.mark.parametrize("N,M,ns", [(2, 3, 1), (5, 31, 2), (31, 128, 33), (32, 129, 40), (33, 256, 4865), (64, 100, 9731),
                                    (65, 384, 1217), (12, 512, 2433), (129, 1000, 5), (20, 2000, 3)])
@pytest.mark.parametrize("kind", ["flips", "bonds", "mixed"])
def test_rbm_eloc_batches(cuda, N, M, ns, kind):
    L = lib()
    ops = _ops(kind, N)
    W, b, a = rbm.init_normal(N, M, (N + M) ** -0.5, seed=N + M, visible_bias=True)
    dev, op = Rbm(W, b, a), compiled(ops)
    s = metropolis.init_uniform(ns, N, 3)

    def run(rows):
        out = torch.full((len(rows),), float("nan"), dtype=torch.float64, device="cuda")
        L.call("qgx_rbm_eloc", L.ptr(dev.table), N, M, C.byref(op.struct), L.ptr(pack(rows)), len(rows), L.ptr(out),
               L.stream_ptr())
        return out.cpu().numpy()

    whole = run(s)
    for cut in (1, 2, 3):
        np.testing.assert_array_equal(run(s[:cut]), whole[:cut])
        np.testing.assert_array_equal(run(s[-cut:]), whole[-cut:])
    rows = np.unique(np.linspace(0, ns - 1, 5).astype(int))
    want = oops.local_energy(s[rows], ops, rbm.RBM(W, b, a).log_psi).real
    np.testing.assert_allclose(whole[rows], want, rtol=2e-5, atol=2e-5 * np.abs(want).max())
