"""Kernels laid out for the FP64 pipe's latency: block inverses and substitutions of the FP64
triangular solves at block edges, the energy statistics' four forms, and the bookkeeping of ResConv
local energies with one- and two-site terms."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 127, 129, 200, 257])
def test_triangular_solves_at_block_edges(cuda, n):
    """Residual of S y = f for a well-conditioned S: below 16 n 2^-53 |S| |y| (factor and two solves)."""
    from quantax_gb300 import _lib as L
    rng = np.random.default_rng(n)
    G = rng.normal(size=(n, 2 * n))
    S = G @ G.T / n + np.eye(n)
    f = rng.normal(size=n)
    St, ft = torch.as_tensor(S.copy()).cuda(), torch.as_tensor(f).cuda()
    nb = C.c_int64(0)
    L.call("qgx_solve_workspace_bytes", n, 1, L.SOLVE_SHIFT, C.byref(nb))
    ws = torch.empty(max(nb.value, 256), dtype=torch.uint8, device="cuda")
    y = torch.empty(n, dtype=torch.float64, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    L.call("qgx_sym_solve", L.ptr(St), n, L.ptr(ft), L.SOLVE_SHIFT, 0.0, 0.0, 0.0, 0.0, L.ptr(y), L.ptr(info), L.ptr(ws),
           ws.numel(), L.stream_ptr())
    y = y.cpu().numpy()
    assert int(info.item()) == 0
    assert np.linalg.norm(S @ y - f) <= 16 * n * 2.0 ** -53 * np.linalg.norm(S, 2) * np.linalg.norm(y)


@pytest.mark.parametrize("ns", [1, 2, 31, 1024, 1025, 5000])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
def test_energy_stats_forms(cuda, ns, weighted, cplx):
    """Compensated FP64 sums: 64 roundings of the largest term at most."""
    from quantax_gb300 import _lib as L
    rng = np.random.default_rng(ns)
    E = rng.normal(size=ns) - 40.0 + (1j * rng.normal(size=ns) if cplx else 0)
    w = rng.random(ns) + 0.5 if weighted else np.ones(ns)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x)).cuda()
    er, ei, r = t(E.real), t(E.imag) if cplx else None, t(w) if weighted else None
    stats = torch.empty(3, dtype=torch.float64, device="cuda")
    br, bi = (torch.empty(ns, dtype=torch.float64, device="cuda") for _ in range(2))
    L.call("qgx_energy_stats", L.ptr(er), L.ptr(ei), L.ptr(r), ns, L.ptr(stats), L.ptr(br), L.ptr(bi) if cplx else None,
           L.stream_ptr())
    mean, plain = (E * w).mean(), E.mean()
    var = (np.abs(E - mean) ** 2 * w).mean()
    bar = (E - plain) * np.sqrt(w / ns)
    tol = 64 * 2.0 ** -53 * np.abs(E).max() ** 2 * w.max()
    assert abs(stats[0].item() - mean.real) <= tol and abs(stats[1].item() - mean.imag) <= tol
    assert abs(stats[2].item() - var) <= tol
    assert np.abs(br.cpu().numpy() - bar.real).max() <= tol
    if cplx:
        assert np.abs(bi.cpu().numpy() - bar.imag).max() <= tol


@pytest.mark.parametrize("ns", [1, 3, 37])
@pytest.mark.parametrize("L,cplx", [(4, True), (6, False)])
def test_local_energies_with_mixed_terms(cuda, ns, L, cplx):
    """A transverse and a longitudinal field beside the J1-J2 exchange: one-site flips, two-site
    flips with elements that vanish on aligned spins, and z terms; FP32 convolutions against the
    FP64 oracle within the 1e-5 (relative to the largest) that the ResConv tests state."""
    import quantax_gb300 as qtx
    from oracle import operators as oops, resconv
    qtx.set_default_dtype(np.complex128 if cplx else np.float64)
    n = L * L
    qtx.sites.Square(L)
    H = qtx.operator.Heisenberg(J=[1.0, 0.5], n_neighbor=[1, 2], msr=True)
    for i in range(n):
        H = H + (-0.7) * qtx.operator.sigma_x(i) + (0.3 if i % 3 else -0.2) * qtx.operator.sigma_z(i)
    state = qtx.state.Variational(qtx.model.ResConv(2, 8, out_dtype=np.complex64 if cplx else None, seed=3))
    rng = np.random.default_rng(ns)
    spins = (2 * rng.integers(0, 2, (ns, n)) - 1).astype(np.int8)
    got = H.Oloc(state, spins).cpu().numpy()
    p = state.get_params_flatten().cpu().numpy().astype(np.float64)

    def log_psi(s):
        x = torch.as_tensor(np.asarray(s, np.float64))
        out = resconv.log_psi_torch(torch.as_tensor(p), x, L, 2, 8, complex_out=cplx)
        return out.numpy()

    want = oops.local_energy(spins, H.op_list, log_psi)
    want = want if cplx else want.real
    qtx.set_default_dtype(np.float64)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("ns", [255, 256, 512, 513, 2048, 2049, 20011])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("cplx", [False, True])
def test_energy_stats_one_cta_or_cluster(cuda, ns, weighted, cplx):
    test_energy_stats_forms(cuda, ns, weighted, cplx)
