"""What the speed of this library is measured on: the work of a variational Monte Carlo run, called
as a user's program calls it (samplers, local energies, log-derivatives, SR / MinSR steps).

A case is a dict of plain values; its "kind" names the call:

  rbm_iteration  one whole iteration of an RBM state: sweep, step, update
  rbm_sweep      one Metropolis sweep of an RBM state
  rbm_eloc       local energies of an RBM state on given samples
  rbm_step       one SR / MinSR step of an RBM state on given samples
  conv_sweep     one SpinExchange sweep of a ResConv state
  conv_logpsi    log psi of a ResConv state on given samples
  conv_eloc      local energies of a ResConv state on given samples
  conv_obar      centred log-derivatives of a ResConv state on given samples
  conv_step      one SR / MinSR step of a ResConv state on given samples
  solve          the MinSR solve alone, on a given Obar and Ebar

RBM states live on the transverse-field Ising chain, ResConv states on the J1-J2 square lattice in
its Sz = 0 sector. Parameters, configurations and matrices come from the seed through numpy and
torch, so `exact` can form the same results in 64 bits without the library.
"""
import math

import numpy as np
import torch

import quantax_gb300 as qtx

ASHIFT = 1e-4  # diagonal shift of the shift solvers
RSHIFT = 1e-6  # their default relative shift


# ---- the cases -------------------------------------------------------------------------------
def listed():
    return [
        # the smallest run, the 8-site chain of the examples: latency of launches and host calls
        {"name": "tfim8_iteration", "kind": "rbm_iteration", "L": 8, "M": 16, "ns": 64, "steps": 8},
        # the sampler of the 64-site chain at 8192 chains, one proposal per site
        {"name": "tfim64_sweep", "kind": "rbm_sweep", "L": 64, "M": 256, "ns": 8192, "steps": 64},
        # local energies of a long chain with a wide RBM, as a serving job has them
        {"name": "tfim128_eloc", "kind": "rbm_eloc", "L": 128, "M": 512, "ns": 4096},
        # the MinSR step of the 64-site chain: 8192 samples, 16640 parameters, FP64 solve
        {"name": "tfim64_minsr_step", "kind": "rbm_step", "L": 64, "M": 256, "ns": 8192, "gram": "3xtf32",
         "solver": "shift"},
        # more samples than parameters (S-path), default arithmetic, odd sizes everywhere
        {"name": "tfim31_sr_step", "kind": "rbm_step", "L": 31, "M": 33, "ns": 4099, "gram": "fp32",
         "solver": "shift"},
        # the 4x4 tutorial's step: real ResConv(2, 8), 1024 samples, every option at its default
        # (FP32 Gram, FP64 pseudo-inverse)
        {"name": "square4_default_step", "kind": "conv_step", "L": 4, "B": 2, "C": 8, "cplx": False, "ns": 1024,
         "conv": "fp32", "gram": "fp32", "solver": "pinv"},
        # the plain method's sweep on the 10x10 square: two proposals per site, FP32 convolutions
        {"name": "square10_sweep", "kind": "conv_sweep", "L": 10, "B": 8, "C": 16, "cplx": True, "ns": 8192,
         "steps": 200, "conv": "fp32"},
        # its local energies: every configuration connected by the J1 and J2 bonds
        {"name": "square10_eloc", "kind": "conv_eloc", "L": 10, "B": 8, "C": 16, "cplx": True, "ns": 1024,
         "conv": "fp32"},
        # the same in the precision form, BF16 convolutions on the tensor cores
        {"name": "square10_eloc_bf16", "kind": "conv_eloc", "L": 10, "B": 8, "C": 16, "cplx": True, "ns": 2048,
         "conv": "bf16"},
        # log-derivatives by the backward pass (always FP32), centred: the matrix of the MinSR step
        {"name": "square10_obar", "kind": "conv_obar", "L": 10, "B": 8, "C": 16, "cplx": True, "ns": 1024},
        # the largest: the Gram and the FP64 solve of 16384 complex samples (32768 stacked rows)
        {"name": "square10_minsr_solve", "kind": "solve", "rows": 32768, "cols": 34944, "gram": "3xtf32",
         "precision": "fp64"},
        # a step of a mid-size serving job: narrow network, BF16 convolutions and Gram, FP64 solve
        {"name": "square6_job_step", "kind": "conv_step", "L": 6, "B": 5, "C": 12, "cplx": True, "ns": 2048,
         "conv": "bf16", "gram": "bf16", "solver": "shift"},
    ]


def draw(rng):
    def spread(lo, hi):  # whole numbers, even over the logarithm
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["rbm_iteration", "rbm_sweep", "rbm_eloc", "rbm_step", "conv_sweep", "conv_logpsi", "conv_eloc",
                       "conv_obar", "conv_step", "solve"])
    if kind.startswith("rbm"):
        L = spread(8, 128)
        c = {"kind": kind, "L": L, "M": min(512, max(8, int(L * rng.choice([1, 2, 4])) + rng.choice([0, 0, 1, -3]))),
             "ns": spread(64, 8192)}
        if kind in ("rbm_iteration", "rbm_sweep"):
            c["steps"] = int(L * rng.choice([1, 2]))
        if kind == "rbm_iteration":
            c["ns"] = min(c["ns"], 2048)
        if kind == "rbm_step":
            c["ns"] = min(c["ns"], 6000)
            c["gram"] = rng.choice(["fp32", "tf32", "bf16", "3xtf32"])
            c["solver"] = "shift"
        return c
    if kind == "solve":
        rows = spread(256, 12000)
        return {"kind": kind, "rows": rows, "cols": max(rows + rng.randint(1, 40), spread(1000, 35000)),
                "gram": rng.choice(["3xtf32", "3xtf32", "tf32", "bf16", "fp32"]),
                "precision": rng.choice(["fp64", "fp64", "mixed"])}
    L = rng.choice([4, 6, 8, 10])
    c = {"kind": kind, "L": L, "B": rng.randint(2, 8), "C": rng.choice([8, 12, 16]), "cplx": rng.random() < 0.7}
    if kind == "conv_obar":
        return dict(c, ns=spread(64, 2048))
    c["conv"] = rng.choice(["fp32", "fp32", "tf32", "bf16"])
    if kind == "conv_sweep":
        return dict(c, ns=spread(256, 8192), steps=spread(8, 2 * L * L))
    if kind == "conv_logpsi":
        return dict(c, ns=spread(64, 65536))
    if kind == "conv_eloc":
        return dict(c, ns=spread(64, 2048))
    return dict(c, ns=spread(256, 2048), gram=rng.choice(["fp32", "3xtf32", "bf16", "tf32"]), solver="shift")


# ---- inputs ----------------------------------------------------------------------------------
def _rng(seed, what):
    return np.random.default_rng([int(seed) & 0xFFFFFFFF, what])


def _rbm_params(case, seed):
    """W (M, N), b (M), a (N), N(0, 0.05^2) float32: the size that the weights have early in training."""
    r = _rng(seed, 1)
    return tuple(r.normal(0.0, 0.05, s).astype(np.float32) for s in ((case["M"], case["L"]), case["M"], case["L"]))


def _conv_params(case, seed):
    """ResConv parameters in the library's flat order: He-normal kernels, small biases."""
    r, parts = _rng(seed, 2), []
    for b in range(case["B"]):
        for layer in range(2):
            cin = 1 if b == 0 and layer == 0 else case["C"]
            parts.append(r.normal(0.0, math.sqrt(2.0 / (9 * cin)), case["C"] * cin * 9))
            if not (layer == 1 and b == case["B"] - 1):
                parts.append(r.normal(0.0, 0.02, case["C"]))
    return np.concatenate(parts).astype(np.float32)


def _spins(case, seed):
    """Random +-1 configurations: uniform on the chain, half filled on the square."""
    r = _rng(seed, 3)
    if case["kind"].startswith("rbm"):
        return (2 * r.integers(0, 2, (case["ns"], case["L"])) - 1).astype(np.int8)
    n = case["L"] ** 2
    base = np.where(np.arange(n) < n // 2, 1, -1).astype(np.int8)
    return r.permuted(np.tile(base, (case["ns"], 1)), axis=1)


def _solve_inputs(case, seed):
    """Obar: rows of a few strong directions over weaker noise, centred and scaled as
    (O - <O>) / sqrt(Ns) is, row stride padded to 8 floats; Ebar: centred, FP64."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    rows, cols = case["rows"], case["cols"]
    buf = torch.zeros((rows, (cols + 7) // 8 * 8), dtype=torch.float32, device="cuda")
    A = buf[:, :cols]
    k = 64
    left = torch.randn((rows, k), generator=g, device="cuda") * torch.logspace(0, -2, k, device="cuda")
    A.normal_(generator=g)
    A.mul_(0.1).addmm_(left, torch.randn((k, cols), generator=g, device="cuda"))
    A.sub_(A.mean(dim=0)).mul_(1.0 / math.sqrt(rows))
    b = torch.randn(rows, generator=g, device="cuda", dtype=torch.float64)
    return A, (b - b.mean()) / math.sqrt(rows)


def _solver(name):
    if name == "pinv":
        return None  # the optimizer's default
    return qtx.optimizer.auto_shift_eig(ashift=ASHIFT)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    qtx.set_random_seed(int(seed) % (1 << 31))
    if s.kind == "solve":
        qtx.set_default_dtype(np.float64)
        qtx.sites.Chain(8)
        owner = qtx.state.Variational(qtx.model.RBM_Dense(8, seed=0))  # holds the solver's workspaces
        s.opt = qtx.optimizer.QNGD(owner, gram=case["gram"], solver=qtx.optimizer.minnorm_shift_eig(
            ashift=ASHIFT, precision=case["precision"]))
        s.A, s.b = _solve_inputs(case, seed)
        return s
    spins = _spins(case, seed)
    if s.kind.startswith("rbm"):
        qtx.set_default_dtype(np.float64)
        qtx.sites.Chain(case["L"])
        s.H = qtx.operator.Ising(h=1.0)
        W, b, a = _rbm_params(case, seed)
        small = s.kind == "rbm_iteration"  # the small runs carry the visible bias
        s.state = qtx.state.Variational(qtx.model.RBM_Dense.from_arrays(W, b, a if small else None))
        if s.kind in ("rbm_iteration", "rbm_sweep"):
            s.sampler = qtx.sampler.LocalFlip(s.state, case["ns"], thermal_steps=0, sweep_steps=case["steps"],
                                              initial_spins=spins)
        else:
            s.samples = qtx.sampler.Samples.from_spins(spins)
        s.opt = qtx.optimizer.SR(s.state, s.H, solver=_solver(case.get("solver")) or _solver("shift"),
                                 gram=case.get("gram", "fp32"))
        return s
    L, n = case["L"], case["L"] ** 2
    qtx.set_default_dtype(np.complex128 if case["cplx"] else np.float64)
    qtx.sites.Square(L, Nparticles=(n // 2, n // 2))
    model = qtx.model.ResConv(case["B"], case["C"], out_dtype=np.complex64 if case["cplx"] else None,
                              conv_precision=case.get("conv", "fp32"), seed=0)
    s.state = qtx.state.Variational(model)
    s.state.set_params(_conv_params(case, seed))
    if s.kind == "conv_sweep":
        s.sampler = qtx.sampler.SpinExchange(s.state, case["ns"], thermal_steps=0, sweep_steps=case["steps"],
                                             initial_spins=spins)
        return s
    s.samples = qtx.sampler.Samples.from_spins(spins)
    if s.kind in ("conv_eloc", "conv_step"):
        s.H = qtx.operator.Heisenberg(J=[1.0, 0.5], n_neighbor=[1, 2], msr=True)
        s.H.compiled()
    if s.kind == "conv_step":
        s.opt = qtx.optimizer.SR(s.state, s.H, solver=_solver(case["solver"]), gram=case["gram"])
    return s


# ---- one pass --------------------------------------------------------------------------------
def run(s):
    if s.kind == "rbm_iteration":
        samples = s.sampler.sweep()
        step = s.opt.get_step(samples)
        s.state.update(1e-2 * step)
        return [samples.packed, samples.log_psi, s.opt.stats, step, s.state.params]
    if s.kind in ("rbm_sweep", "conv_sweep"):
        samples = s.sampler.sweep()
        return [samples.packed, samples.log_psi, s.sampler.accepts]
    if s.kind in ("rbm_eloc", "conv_eloc"):
        return s.H.Oloc(s.state, s.samples)
    if s.kind == "conv_logpsi":
        return s.state.log_psi_packed(s.samples.packed)
    if s.kind == "conv_obar":
        return list(s.state.obar(s.samples))
    if s.kind == "solve":
        return s.opt.solve(s.A, s.b)
    step = s.opt.get_step(s.samples)
    return [step, s.opt.stats]


# ---- the work a pass cannot do without -------------------------------------------------------
def _conv_flops(case):
    """One forward: multiply and add of every 3x3 convolution."""
    return 2.0 * case["L"] ** 2 * 9 * case["C"] * (1 + (2 * case["B"] - 1) * case["C"])


def _conv_nparams(case):
    return sum(case["C"] * (1 if b == 0 else case["C"]) * 9 + case["C"] ** 2 * 9 + 2 * case["C"]
               for b in range(case["B"])) - case["C"]


def _solve_work(rows, cols):
    """Gram of the shorter side (its symmetric half), Cholesky, two triangular solves, projection."""
    n, k = min(rows, cols), max(rows, cols)
    return {"bytes": 4.0 * rows * cols + 8.0 * (rows + cols), "flops": float(n) * n * k + n ** 3 / 3.0 + 2.0 * n * n
            + 2.0 * rows * cols}


def work(case):
    kind = case["kind"]
    if kind == "solve":
        return _solve_work(case["rows"], case["cols"])
    ns, L = case["ns"], case["L"]
    if kind.startswith("rbm"):
        M = case["M"]
        npar = M * L + M
        forward, ratio = 2.0 * M * L, 4.0 * M  # theta = W s + b; one flip's ratio from theta
        sweep = {"bytes": 4.0 * npar + ns * (2.0 * L / 8 + 8), "flops": ns * (forward + case.get("steps", 0) * ratio)}
        eloc = {"bytes": 4.0 * npar + ns * (L / 8.0 + 8), "flops": ns * (forward + L * ratio)}
        solve = _solve_work(ns, npar)
        if kind == "rbm_sweep":
            return sweep
        if kind == "rbm_eloc":
            return eloc
        # Obar is an intermediate of the step; samples in, step out
        step = {"bytes": eloc["bytes"] + 8.0 * npar, "flops": eloc["flops"] + 2.0 * ns * npar + solve["flops"]}
        if kind == "rbm_step":
            return step
        return {k: sweep[k] + step[k] for k in step}
    npar, fwd, words = _conv_nparams(case), _conv_flops(case), (L * L + 31) // 32
    cot = 2 if case["cplx"] else 1
    changed = (L * L / 2) / (L * L - 1.0)  # share of exchange proposals whose spins differ
    conn = 4 * L * L * changed  # antiparallel pairs among the 2 N + 2 N bonds
    if kind == "conv_sweep":
        return {"bytes": 4.0 * npar + ns * (8.0 * words + 12), "flops": ns * fwd * (1 + changed * case["steps"])}
    if kind == "conv_logpsi":
        return {"bytes": 4.0 * npar + ns * (4.0 * words + 8), "flops": ns * fwd}
    eloc = {"bytes": 4.0 * npar + ns * (4.0 * words + 8 * cot), "flops": ns * fwd * (1 + conn)}
    if kind == "conv_eloc":
        return eloc
    rows = cot * ns
    obar = {"bytes": 4.0 * npar + 4.0 * ns * words + 4.0 * rows * npar, "flops": ns * fwd * (1 + 2 * cot)
            + 2.0 * rows * npar}
    if kind == "conv_obar":
        return obar
    solve = _solve_work(rows, npar)
    return {"bytes": eloc["bytes"] + 8.0 * npar, "flops": eloc["flops"] + obar["flops"] + solve["flops"]}


# ---- the same results in 64 bits, in plain torch ----------------------------------------------
def _t(a):
    return torch.as_tensor(a, dtype=torch.float64, device="cuda")


def _logcosh(x):
    x = x.abs()
    return x + torch.log1p(torch.exp(-2 * x)) - math.log(2.0)


def _rbm_log_psi(p, s):
    W, b, _ = p
    return _logcosh(s @ W.T + b).sum(1)


def _rbm_eloc(p, s):
    L = s.shape[1]
    e = -(s * s.roll(-1, 1)).sum(1)  # -J sum s_i s_(i+1), periodic
    theta = s @ p[0].T + p[1]
    here = _logcosh(theta).sum(1)
    for k in range(L):
        e -= torch.exp(_logcosh(theta - 2 * s[:, k:k + 1] * p[0][:, k]).sum(1) - here)
    return e


def _conv_weights(flat, case):
    out, at, C = [], 0, case["C"]
    for b in range(case["B"]):
        for layer in range(2):
            cin = 1 if b == 0 and layer == 0 else C
            w = flat[at:at + C * cin * 9].reshape(C, cin * 9)
            at += C * cin * 9
            if layer == 1 and b == case["B"] - 1:
                bias = torch.zeros(C, dtype=flat.dtype, device=flat.device)
            else:
                bias = flat[at:at + C]
                at += C
            out.append((w, bias))
    return out


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _conv(x, w, bias):
    """3x3 periodic cross-correlation of x (channels, batch, L, L)."""
    taps = torch.stack([x.roll((1 - dy, 1 - dx), (2, 3)) for dy in range(3) for dx in range(3)], 1)
    y = w @ taps.reshape(taps.shape[0] * 9, -1) + bias[:, None]
    return y.reshape(w.shape[0], *x.shape[1:])


def _conv_log_psi(flat, s, case):
    """(Re, Im) of log psi of s (batch, N)."""
    L, C, B = case["L"], case["C"], case["B"]
    ws = _conv_weights(flat, case)
    x = s.reshape(1, -1, L, L)
    for b in range(B):
        h = x / math.sqrt(b + 1)
        h = h / math.sqrt(2.0) if b == 0 else _gelu(h)
        x = _conv(_gelu(_conv(h, *ws[2 * b])), *ws[2 * b + 1]) + (x.expand(C, -1, L, L) if b == 0 else x)
    z = (x / math.sqrt(B + 1)).transpose(0, 1).reshape(s.shape[0], C, L * L)
    re = (z[:, :C // 2] if case["cplx"] else z).reshape(s.shape[0], -1)
    im = z[:, C // 2:].reshape(s.shape[0], -1) if case["cplx"] else torch.zeros_like(re)
    m = re.max(1, keepdim=True).values
    sr, si = (torch.exp(re - m) * torch.cos(im)).sum(1), (torch.exp(re - m) * torch.sin(im)).sum(1)
    return m[:, 0] + 0.5 * torch.log(sr * sr + si * si) - math.log(re.shape[1]), torch.atan2(si, sr)


def _chunked_log_psi(flat, s, case, chunk=8192):
    parts = [torch.stack(_conv_log_psi(flat, c, case), 1) for c in s.split(chunk)]
    return torch.cat(parts)


def _square_bonds(L):
    """(i, j, J, sign) of the J1 (sign -1: Marshall rule) and J2 = 0.5 bonds, each once."""
    out = []
    for y in range(L):
        for x in range(L):
            for dy, dx, J, sign in ((0, 1, 1.0, -1.0), (1, 0, 1.0, -1.0), (1, 1, 0.5, 1.0), (1, -1, 0.5, 1.0)):
                out.append((y * L + x, (y + dy) % L * L + (x + dx) % L, J, sign))
    return out


def _conv_eloc(flat, s, case):
    bonds = _square_bonds(case["L"])
    i, j = (torch.tensor([b[k] for b in bonds], device="cuda") for k in (0, 1))
    J, sign = (_t([b[k] for b in bonds]) for k in (2, 3))
    zz = s[:, i] * s[:, j]
    lp = _chunked_log_psi(flat, s, case)
    re, im = (J * zz).sum(1), torch.zeros(s.shape[0], dtype=torch.float64, device="cuda")
    who, which = torch.nonzero(zz < 0, as_tuple=True)
    for a in range(0, len(who), 65536):
        w, q = who[a:a + 65536], which[a:a + 65536]
        c = s[w].clone()
        rows = torch.arange(len(w), device="cuda")
        c[rows, i[q]], c[rows, j[q]] = s[w, j[q]], s[w, i[q]]
        d = _chunked_log_psi(flat, c, case) - lp[w]
        amp = 2 * (J * sign)[q] * torch.exp(d[:, 0])
        re.index_add_(0, w, amp * torch.cos(d[:, 1]))
        im.index_add_(0, w, amp * torch.sin(d[:, 1]))
    return torch.complex(re, im) if case["cplx"] else re


def _conv_jacobian(flat, s, case, chunk=64):
    """Rows [Re O; Im O] (Re only for real output)."""
    def part(k):
        g = torch.func.grad(lambda p, x: _conv_log_psi(p, x[None], case)[k][0])
        f = torch.func.vmap(g, (None, 0))
        return torch.cat([f(flat, c) for c in s.split(chunk)])

    return torch.cat([part(0), part(1)]) if case["cplx"] else part(0)


def _centre(O, ns):
    """(Obar, Omean) of O's one or two blocks of ns rows."""
    blocks = O.split(ns)
    means = [b.mean(0) for b in blocks]
    return torch.cat([(b - m) / math.sqrt(ns) for b, m in zip(blocks, means)]), means


def _step(A, b):
    """The shifted MinSR (fewer rows than columns) or SR solve."""
    if A.shape[0] < A.shape[1]:
        M, back = A @ A.T, lambda y: A.T @ y
    else:
        M, back, b = A.T @ A, (lambda y: y), A.T @ b
    M.diagonal().add_(RSHIFT * float(torch.trace(M)) + ASHIFT)
    return back(torch.cholesky_solve(b[:, None], torch.linalg.cholesky(M))[:, 0])


def _energy(E, ns):
    """(stats, Ebar) of local energies E."""
    re, im = (E.real, E.imag) if E.is_complex() else (E, torch.zeros_like(E))
    mr, mi = re.mean(), im.mean()
    var = ((re - mr) ** 2 + (im - mi) ** 2).mean()
    bar = torch.cat([re - mr, im - mi]) if E.is_complex() else re - mr
    return torch.stack([mr, mi, var]), bar / math.sqrt(ns)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("rbm_iteration", "rbm_sweep", "conv_sweep"):
        return None  # the chains follow accept decisions taken on 32-bit amplitudes
    if kind == "solve":
        rows, cols = case["rows"], case["cols"]
        if float(rows) * rows * (cols + rows / 3) > 1.5e12:
            return None
        A, b = _solve_inputs(case, seed)
        return _step(A.double(), b)
    s = _t(_spins(case, seed))
    ns = case["ns"]
    if kind.startswith("rbm"):
        p = [_t(x) for x in _rbm_params(case, seed)]
        E = _rbm_eloc(p, s)
        if kind == "rbm_eloc":
            return E
        th = torch.tanh(s @ p[0].T + p[1])
        O = torch.cat([(th[:, :, None] * s[:, None, :]).reshape(ns, -1), th], 1)
    else:
        flat = _t(_conv_params(case, seed))
        if kind == "conv_logpsi":
            lp = _chunked_log_psi(flat, s, case)
            return torch.complex(lp[:, 0], lp[:, 1]) if case["cplx"] else lp[:, 0]
        if kind == "conv_obar":
            O = _conv_jacobian(flat, s, case)
            A, means = _centre(O, ns)
            return [A, torch.complex(*means) if case["cplx"] else means[0]]
        if kind == "conv_eloc":
            return _conv_eloc(flat, s, case)
        E = _conv_eloc(flat, s, case)
        O = _conv_jacobian(flat, s, case)
    stats, bar = _energy(E, ns)
    if case["solver"] == "pinv" or float(ns) ** 2 * O.shape[1] > 3e12:
        # the pseudo-inverse's cut-off sits at FP32 resolution: its step has no 64-bit value
        return [None, stats]
    return [_step(_centre(O, ns)[0], bar), stats]
