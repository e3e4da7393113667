"""RBM local energies with tables at the limit of shared memory: staged whole up to it, read from
device memory past it. Sizes on both sides, one by one and in a batch; agreement with the FP64 oracle
within 2e-5 of the largest (FP32 log ratios), and the same bits in both calls."""
import ctypes as C

import numpy as np
import pytest
import torch

from oracle import lattice, metropolis, operators as oops, rbm
from test_gpu_rbm import Rbm, compiled, lib, pack

pytestmark = pytest.mark.gpu

# (N, M): the last that fit 227 KB (3 N padded M + padded M + N floats), and the next
FIT = [(147, 128), (148, 120), (150, 128), (74, 256), (75, 200), (50, 384)]
PAST = [(151, 128), (76, 256), (51, 384)]


def job(N, M, ns):
    ops = oops.chain_tfim(N, h=0.7, J=1.2)
    W, b, a = rbm.init_normal(N, M, (N + M) ** -0.5, seed=N + M, visible_bias=True)
    s = metropolis.init_uniform(ns, N, 3)
    return ops, rbm.RBM(W, b, a), Rbm(W, b, a), compiled(ops), s, pack(s)


def batched(jobs):
    L = lib()
    outs = [torch.full((len(j[4]),), float("nan"), dtype=torch.float64, device="cuda") for j in jobs]
    descs = (L.RbmElocJob * len(jobs))()
    for d, (_, net, dev, op, s, packed), out in zip(descs, jobs, outs):
        d.table, d.n, d.m, d.op = L.ptr(dev.table), s.shape[1], net.W.shape[0], C.pointer(op.struct)
        d.spins, d.ns, d.eloc = L.ptr(packed), len(s), L.ptr(out)
    launches = C.c_int32(-1)
    L.call("qgx_rbm_eloc_batched", descs, len(jobs), C.byref(launches), L.stream_ptr())
    return [o.cpu().numpy() for o in outs], launches.value


@pytest.mark.parametrize("N,M", FIT + PAST)
@pytest.mark.parametrize("ns", [3, 5000])
def test_tables_beside_the_limit(cuda, N, M, ns):
    L = lib()
    j = job(N, M, ns)
    ops, net, dev, op, s, packed = j
    out = torch.full((ns,), float("nan"), dtype=torch.float64, device="cuda")
    L.call("qgx_rbm_eloc", L.ptr(dev.table), N, M, C.byref(op.struct), L.ptr(packed), ns, L.ptr(out), L.stream_ptr())
    got = out.cpu().numpy()
    rows = np.unique(np.linspace(0, ns - 1, 4).astype(int))
    want = oops.local_energy(s[rows], ops, net.log_psi).real
    np.testing.assert_allclose(got[rows], want, rtol=2e-5, atol=2e-5 * np.abs(want).max())
    (again,), _ = batched([j])
    np.testing.assert_array_equal(again, got)


@pytest.mark.parametrize("small,edge,past", [((20, 128), (150, 128), (151, 128)), ((10, 256), (75, 256), (76, 256)),
                                             ((5, 384), (50, 384), (51, 384))])
def test_staged_jobs_share_a_launch(cuda, small, edge, past):
    """A batch launches once for its staged tables of a width and once for the others: the largest
    table that fits is a staged one."""
    jobs = [job(*small, 7), job(*edge, 9)]
    assert batched(jobs)[1] == 1
    assert batched(jobs + [job(*past, 4)])[1] == 2
