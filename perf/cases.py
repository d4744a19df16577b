"""Performance cases: the work that users of conatus_gb300 have it do, through its entry points.

A case is a dict of plain values. ``prepare`` makes what a user's program holds before the call (the
problem, its device plan and factorizations, the inputs, on the GPU unless the call takes host
arrays), ``run`` makes one pass, ``work`` says what a pass cannot do without, and ``exact`` gives a
pass's outputs in 64 bits with plain torch and numpy from the committed problem data (dense solves,
matrix and library transforms), where that takes seconds.
"""
from __future__ import annotations

import json
import math
import os

import numpy as np
import torch

from conatus_gb300 import _lib, core
from conatus_gb300 import workloads as W
from conatus_gb300.ensemble import FourierEnsemble, ks_members
from conatus_gb300.ivp import DeviceProblem, IVPSolver
from conatus_gb300.template import GroupedProblem, StackedProblem

C128 = torch.complex128
PROBLEMS = os.path.join(os.path.dirname(os.path.abspath(W.__file__)), "problems")
LX_RB = 2 * math.pi / 3.117            # period of the Rayleigh-Benard boxes


# ------------------------------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the headline configuration's step (plane channel, SBDF3) at half its Fourier resolution:
        # a trajectory from a given state, start-up and finite-state check included
        dict(name="channel_step", kind="step", problem="channel", nx=96, nz=96, scheme="SBDF3", dt=5e-3,
             precision="fp64", steps=8),
        # the same in the FP32 form, chosen by users who trade accuracy for rate
        dict(name="channel_step_fp32", kind="step", problem="channel", nx=96, nz=96, scheme="SBDF3", dt=5e-3,
             precision="fp32", steps=8),
        # 2D Rayleigh-Benard at the reference's published size and scheme: launches and latency count
        dict(name="rb_rk443", kind="step", problem="rb_nz64", nx=256, nz=0, scheme="RK443", dt=1e-4,
             precision="fp64", steps=10),
        # 1D Burgers: the smallest problem, one system, a long run of tiny steps
        dict(name="burgers_run", kind="step", problem="burgers_n128", nx=0, nz=0, scheme="SBDF2", dt=1e-4,
             precision="fp64", steps=50),
        # the explicit right-hand side at the headline configuration's full size (192 x 129 x 192)
        dict(name="channel_rhs", kind="rhs", problem="channel", nx=192, nz=192, precision="fp64"),
        # the implicit solves of a step (every bucket) at two thirds of the headline resolution
        dict(name="channel_solve", kind="solve", problem="channel", nx=128, nz=128, a=11 / 6 / 5e-3,
             precision="fp64"),
        # the Fourier and Chebyshev transforms by themselves, both directions, ragged lengths
        dict(name="transforms", kind="transforms", fields=3, nx=90, nz=100, ny=97),
        # a serving pool: two Rayleigh-Benard requests of one resolution stepped together
        dict(name="rb_pool", kind="ensemble", nzs="48", cases=2, scheme="SBDF2", precision="fp64", steps=20),
        # an ensemble of Rayleigh-Benard cases of three resolutions in the FP32 form
        dict(name="rb_ensemble_fp32", kind="ensemble", nzs="32,48,64", cases=48, scheme="SBDF2",
             precision="fp32", steps=10),
        # the Kuramoto-Sivashinsky ensemble: uneven members, one fused launch per step
        dict(name="ks_ensemble", kind="ks", members=4096, precision="fp32", steps=20),
        # the reference's GPU core: its batched complex factors solving on caller-owned device memory
        dict(name="core_device", kind="core", where="device", dtype="z", problem="rb_nz64", batch=128,
             transpose=False),
        # the reference's CPU core: real factors, host arrays in and out of every solve
        dict(name="core_host", kind="core", where="host", dtype="d", problem="rb_nz32_ra", batch=31,
             transpose=False),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "rhs", "rhs", "solve", "solve", "transforms", "ensemble", "ks", "core"])
    precision = rng.choice(["fp64", "fp64", "fp64", "fp32"])
    if kind in ("step", "rhs", "solve"):
        family = rng.choice(["channel", "rb", "burgers"])
        case = dict(kind=kind, nx=0, nz=0, precision=precision)
        if family == "channel":
            top = {"step": 96, "rhs": 192, "solve": 128}[kind]
            case.update(problem="channel", nx=_even(rng, 16, top), nz=_even(rng, 16, top))
        elif family == "rb":
            case.update(problem="rb_nz%s" % rng.choice(["64", "32_ra", "48_ra", "80_ra", "96_ra"]),
                        nx=_even(rng, 32, 512))
        else:
            case.update(problem="burgers_n%d_nu" % (32 * rng.randint(2, 16)))
        if kind == "step":
            scheme = rng.choice(["SBDF1", "SBDF2", "SBDF3", "SBDF4", "CNAB2", "RK222", "RK443"])
            steps = rng.randint(4, 6) if family == "channel" else rng.randint(5, 12)
            case.update(scheme=scheme, dt=5e-3 if family == "channel" else 2e-5, steps=steps)
        elif kind == "solve":
            case.update(a=rng.choice([1.0, 1.5, 11 / 6]) / (5e-3 if family == "channel" else 1e-4))
        return case
    if kind == "transforms":
        return dict(kind=kind, fields=rng.randint(1, 8), nx=_even(rng, 8, 192), nz=_even(rng, 8, 192),
                    ny=_log(rng, 12, 200))
    if kind == "ensemble":
        nzs = rng.choice(["32", "48", "64", "80", "96", "32,48", "32,48,64", "48,96"])
        return dict(kind=kind, nzs=nzs, cases=_log(rng, 2, 24), scheme=rng.choice(["SBDF2", "RK222"]),
                    precision=precision, steps=rng.randint(5, 10))
    if kind == "ks":
        return dict(kind=kind, members=_log(rng, 16, 4096), precision=precision, steps=rng.randint(5, 20))
    problem = rng.choice(["rb_nz32_ra", "rb_nz48_ra", "rb_nz64", "rb_nz96_ra", "channel_ny17"])
    return dict(kind="core", where=rng.choice(["device", "host"]), dtype=rng.choice(["z", "d"]), problem=problem,
                batch=_log(rng, 1, 128), transpose=rng.random() < 0.3)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(rng, lo, hi):
    return 2 * _log(rng, lo // 2, hi // 2)


# ------------------------------------------------------------------------------------------------
# what a user has in hand

def _template(name):
    return W.load_template("channel_ny129" if name == "channel" else name)


def _problem(case):
    """The problem of a step, rhs or solve case (Ra and nu of the parametric templates: ordinary ones)."""
    tpl = _template(case["problem"])
    params = {"Ra": 1e5, "nu": 0.01 / math.pi}
    params = {k: params[k] for k in tpl.linear_params} or None
    return tpl.instantiate([n for n in (case["nx"], case["nz"]) if n] or None, None, params)


def _state(case, P, seed):
    """A seeded initial state of the workload (per bucket, on the host)."""
    if case["problem"] == "channel":
        return W.channel_state(P, seed)
    if case["problem"].startswith("rb"):
        return W.rayleigh_benard_state(P, seed)
    C = W.burgers_state(P)
    rng = np.random.default_rng(seed)
    b = P.tpl.buckets[0]
    pos = [i for n in range(12) for i, (v, c, m) in enumerate(b.col) if m == n]
    bump = np.zeros(len(pos))
    for k in range(4):                     # T_{k+2} - T_k vanishes at both walls
        g = 0.1 * rng.standard_normal()
        bump[k + 2] += g
        bump[k] -= g
    C[0][0, pos] += bump
    return C


def _smooth(case, seed):
    """Spectra that fall off in every direction, as resolved fields do (per bucket, on the host)."""
    spec = _Spec(case["problem"])
    rng = np.random.default_rng(seed)
    out = []
    for b, (modes, _) in zip(spec.buckets, spec.systems(case["nx"], case["nz"])):
        k2 = 1.0 + np.sum(np.asarray(modes, float) ** 2, axis=1)
        n = np.maximum(b["col"][:, 2], 0).astype(float)
        fall = 0.3 * (k2 ** -0.8)[:, None] * ((1.0 + n) ** -1.5)[None, :]
        z = rng.standard_normal((2,) + fall.shape)
        out.append((z[0] + (0 if b["kind"] == "real" else 1j) * z[1]) * fall)
    return out


def _rhs_rows(case, seed):
    """Right-hand sides of the implicit solves: rows as a step hands them over."""
    spec = _Spec(case["problem"])
    rng = np.random.default_rng(seed)
    out = []
    for b, (modes, _) in zip(spec.buckets, spec.systems(case["nx"], case["nz"])):
        k2 = 1.0 + np.sum(np.asarray(modes, float) ** 2, axis=1)
        n = np.maximum(b["row"][:, 2], 0).astype(float)
        fall = (k2 ** -0.8)[:, None] * ((1.0 + n) ** -1.5)[None, :]
        fall[:, : b["r"]] = 0.0             # homogeneous boundary rows
        z = rng.standard_normal((2,) + fall.shape)
        out.append((z[0] + (0 if b["kind"] == "real" else 1j) * z[1]) * fall)
    return out


def _stack(case, seed):
    """Rayleigh-Benard cases spread over the resolutions ``nzs``, Ra log-uniform: the problem, the
    stacked state, the time step (an advective limit) and per resolution (nz, Ra of its cases, states)."""
    rng = np.random.default_rng(seed)
    nzs = [int(s) for s in case["nzs"].split(",")]
    stacks, states, parts, dt = [], [], [], 1e-4
    for i, nz in enumerate(nzs):
        count = case["cases"] // len(nzs) + (1 if i < case["cases"] % len(nzs) else 0)
        if count == 0:
            continue
        tpl = W.load_template(f"rb_nz{nz}_ra")
        ra = 10 ** rng.uniform(4, 6, count)
        S = StackedProblem(tpl, [4 * nz], [{"Ra": float(r)} for r in ra])
        st = [W.rayleigh_benard_state(tpl.instantiate([4 * nz], None, {"Ra": float(r)}), seed=seed * 1000 + j)
              for j, r in enumerate(ra)]
        stacks.append(S)
        states.append(S.stack_states(st))
        parts.append((nz, ra, st))
        dt = min(dt, 0.25 * (LX_RB / (4 * nz)) / math.sqrt(float(ra.max())))
    if len(stacks) == 1:
        return stacks[0], states[0], dt, parts
    G = GroupedProblem(stacks)
    return G, G.stack_states(states), dt, parts


def _core_mats(case, seed):
    """(n, border rows, CSR matrices, right-hand sides) of a core case: the systems a M + L of
    consecutive Fourier modes; the real ones hold each complex system as (cos, sin) pairs."""
    spec = _Spec(case["problem"])
    b = spec.buckets[-1]
    d = len(spec.lengths)
    rng = np.random.default_rng(seed)
    j = np.arange(1, case["batch"] + 1)
    kw = 2 * np.pi * np.stack([j / L for L in spec.lengths], axis=1) if d else np.zeros((1, 0))
    M, L = spec.values(b, kw)
    A = M / float(rng.uniform(1e-4, 2e-4)) + L
    n, ip, ix = b["n"], b["indptr"], b["indices"]
    rhs = rng.standard_normal((case["batch"], n)) + 1j * rng.standard_normal((case["batch"], n))
    rhs *= (1.0 + np.maximum(b["row"][:, 2], 0)) ** -1.0
    if case["dtype"] == "z":
        return n, list(range(b["r"])), [(n, ip, ix, a) for a in A], rhs
    rows = np.repeat(np.arange(n), np.diff(ip))
    mats = []
    for a in A:
        r2 = np.concatenate([2 * rows, 2 * rows, 2 * rows + 1, 2 * rows + 1])
        c2 = np.concatenate([2 * ix, 2 * ix + 1, 2 * ix, 2 * ix + 1])
        v2 = np.concatenate([a.real, -a.imag, a.imag, a.real])
        keep = v2 != 0
        order = np.lexsort((c2[keep], r2[keep]))
        p2 = np.concatenate([[0], np.cumsum(np.bincount(r2[keep], minlength=2 * n))])
        mats.append((2 * n, p2.astype(np.int32), c2[keep][order].astype(np.int32), v2[keep][order]))
    flat = np.empty((case["batch"], 2 * n))
    flat[:, 0::2], flat[:, 1::2] = rhs.real, rhs.imag
    return 2 * n, list(range(2 * b["r"])), mats, flat


def _smooth5(n, even=False):
    """The smallest 2^a 3^b 5^c >= n, as grids are chosen."""
    while True:
        k = n
        for p in (2, 3, 5):
            while k % p == 0:
                k //= p
        if k == 1 and not (even and n % 2):
            return n
        n += 1


def _transform_sizes(case):
    nx, nz, ny, f = case["nx"], case["nz"], case["ny"], case["fields"]
    return f, nx // 2, nz, ny, _smooth5(3 * nx // 2), _smooth5(3 * nz // 2), _smooth5(3 * ny // 2, even=True)


def _transform_inputs(case, seed):
    """Coefficients [field][kx][kz][n] and grid values [field][x][z][y], as the right-hand side has them."""
    f, K, nz, ny, mx, mz, my = _transform_sizes(case)
    g = torch.Generator("cuda").manual_seed(seed)
    z = torch.randn((f, K, nz, ny), dtype=C128, device="cuda", generator=g)
    kx = torch.arange(K, device="cuda", dtype=torch.float64).view(1, -1, 1, 1)
    kz = torch.fft.fftfreq(nz, 1 / nz, device="cuda", dtype=torch.float64).view(1, 1, -1, 1)
    n = torch.arange(ny, device="cuda", dtype=torch.float64).view(1, 1, 1, -1)
    z = z * (1 + kx * kx + kz * kz) ** -0.8 * (1 + n) ** -1.5
    z[:, :, nz // 2] = 0                                     # the Nyquist mode is not used
    mirror = torch.remainder(-torch.arange(nz, device="cuda"), nz)
    z[:, 0] = 0.5 * (z[:, 0] + z[:, 0][:, mirror].conj())    # the kx = 0 plane of real fields
    phase = 6.2831853 * torch.rand((f, 3), dtype=torch.float64, device="cuda", generator=g)
    lin = lambda m: torch.arange(m, device="cuda", dtype=torch.float64) * (2 * math.pi / m)
    wave = (torch.sin(lin(mx) + phase[:, :1]).view(f, mx, 1, 1) * torch.cos(2 * lin(mz) + phase[:, 1:2]).view(f, 1, mz, 1)
            * torch.sin(0.5 * lin(my) + phase[:, 2:]).view(f, 1, 1, my))
    grid = wave + 0.1 * torch.randn((f, mx, mz, my), dtype=torch.float64, device="cuda", generator=g)
    return z.contiguous(), grid.contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        P = _problem(case)
        solver = IVPSolver(P, scheme=case["scheme"], dt=case["dt"], precision=case["precision"])
        return dict(kind=kind, solver=solver, X=solver.dev.to_device(_state(case, P, seed)), steps=case["steps"])
    if kind == "ensemble":
        P, st, dt, _ = _stack(case, seed)
        solver = IVPSolver(P, scheme=case["scheme"], dt=dt, precision=case["precision"])
        return dict(kind="step", solver=solver, X=solver.dev.to_device(st), steps=case["steps"])
    if kind == "ks":
        N, L = ks_members(case["members"], seed=0)
        ens = FourierEnsemble(W.load_template("ks"), N, L, scheme="SBDF2", dt=0.01, precision=case["precision"])
        return dict(kind=kind, solver=ens, X=ens.random_state(seed=seed), steps=case["steps"])
    if kind in ("rhs", "solve"):
        dev = DeviceProblem(_problem(case), precision=case["precision"])
        make = _smooth if kind == "rhs" else _rhs_rows
        state = dict(kind=kind, dev=dev, x=dev.to_device(make(case, seed)), out=dev.zeros())
        if kind == "solve":
            state["a"] = case["a"]
            dev.factor(case["a"], 1.0)
            if case["precision"] == "fp32":
                dev.ensure_residual(case["a"], 1.0)
        return state
    if kind == "transforms":
        f, K, nz, ny, mx, mz, my = _transform_sizes(case)
        z, grid = _transform_inputs(case, seed)
        new = lambda shape, dt: torch.zeros(shape, dtype=dt, device="cuda")
        return dict(kind=kind, sizes=(f, K, nz, ny, mx, mz, my), z=z, grid=grid,
                    b1=new((f, K, nz, my), C128), b2=new((f, K, mz, my), C128), b3=new((f, mx, mz, my), torch.float64),
                    f1=new((f, K, mz, my), C128), f2=new((f, K, nz, my), C128), f3=new((f, K, nz, ny), C128))
    n, border, mats, rhs = _core_mats(case, seed)
    if case["where"] == "host":
        cls = core.BorderedBandedBatchZ if case["dtype"] == "z" else core.BorderedBandedBatchD
        return dict(kind="core_host", h=cls(mats, border), b=rhs, transpose=case["transpose"])
    cls = core.cuda.BandedBatchZ if case["dtype"] == "z" else core.cuda.BandedBatchD
    h = cls(mats, border)
    if case["transpose"]:
        h.prepare_transpose()
    b = torch.as_tensor(rhs, device="cuda")
    torch.cuda.synchronize()
    return dict(kind="core_device", h=h, b=b, x=torch.empty_like(b), transpose=case["transpose"])


def run(state):
    kind = state["kind"]
    if kind == "step":
        solver = state["solver"]
        solver.set_state(state["X"])
        solver.run_graph(state["steps"])
        return solver.X
    if kind == "ks":
        ens = state["solver"]
        ens.set_state(state["X"])
        ens.run_graph(state["steps"])
        return ens.X
    if kind == "rhs":
        state["dev"].F(state["x"], state["out"])
        return state["out"]
    if kind == "solve":
        state["dev"].solve(state["a"], 1.0, state["x"], state["out"])
        return state["out"]
    if kind == "transforms":
        f, K, nz, ny, mx, mz, my = state["sizes"]
        s = torch.cuda.current_stream().cuda_stream
        p = lambda name: state[name].data_ptr()
        # coefficients -> grid
        _lib.call("cng_cheb_transform", 0, p("z"), p("b1"), f * K * nz, ny, my, s)
        _lib.call("cng_fft_axis", 0, p("b1"), p("b2"), f * K, my, nz, mz, s)
        _lib.call("cng_rfft_axis", 0, p("b2"), p("b3"), f, mz * my, K, mx, s)
        # grid -> coefficients
        _lib.call("cng_rfft_axis", 1, p("grid"), p("f1"), f, mz * my, K, mx, s)
        _lib.call("cng_fft_axis", 1, p("f1"), p("f2"), f * K, my, nz, mz, s)
        _lib.call("cng_cheb_transform", 1, p("f2"), p("f3"), f * K * nz, ny, my, s)
        return state["b3"], state["f3"]
    if kind == "core_host":
        return state["h"].solve(state["b"], transpose=state["transpose"])
    h, b, x = state["h"], state["b"], state["x"]
    s = torch.cuda.current_stream().cuda_stream
    if state["transpose"]:
        x.copy_(b)
        h.solve_transpose_ptr(x.data_ptr(), x.shape[0], x.shape[1], s)
    else:
        h.solve_mapped_ptr(b.data_ptr(), 0, x.data_ptr(), 0, s)
    return x


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "ks":
        N, _ = ks_members(case["members"], seed=0)
        modes = sum(int(n) // 2 for n in N)
        fl = sum(3 * 2.5 * 1.5 * n * math.log2(1.5 * n) for n in map(int, N))
        return dict(bytes=32.0 * modes, flops=case["steps"] * fl)
    if kind == "transforms":
        f, K, nz, ny, mx, mz, my = _transform_sizes(case)
        fl = f * K * nz * 5 * my * math.log2(my) + f * K * my * 5 * mz * math.log2(mz) \
            + f * mz * my * 2.5 * mx * math.log2(mx)
        return dict(bytes=2.0 * f * (16 * K * nz * ny + 8 * mx * mz * my), flops=2 * fl)
    if kind == "core":
        b = _Spec(case["problem"]).buckets[-1]
        n, nnz = b["n"], len(b["indices"])
        w = 16 if case["dtype"] == "z" else 8
        n, nnz = (n, nnz) if case["dtype"] == "z" else (2 * n, 2 * nnz)
        return dict(bytes=float(case["batch"] * w * (2 * n + nnz)), flops=case["batch"] * (8 if w == 16 else 2) * nnz)
    if kind == "ensemble":
        total = dict(bytes=0.0, flops=0.0)
        nzs = [int(s) for s in case["nzs"].split(",")]
        for nz in nzs:
            one = _step_work(_Spec(f"rb_nz{nz}_ra"), 4 * nz, 0, case)
            total = {k: total[k] + one[k] * case["cases"] / len(nzs) for k in total}
        return total
    spec = _Spec(case["problem"])
    if kind == "step":
        return _step_work(spec, case["nx"], case["nz"], case)
    if kind == "rhs":
        return _rhs_work(spec, case["nx"], case["nz"])
    return _solve_work(spec, case["nx"], case["nz"])


def _rhs_work(spec, nx, nz):
    """The state read and the rows written once; one transform per factor and output."""
    vec = 16.0 * spec.unknowns(nx, nz)
    sizes = [_smooth5(3 * n // 2) for n in (nx, nz) if n] + ([_smooth5(3 * spec.ny // 2)] if spec.ny > 1 else [])
    pts = math.prod(sizes)
    fl = 2.5 * (len(spec.factors) + len(spec.outputs)) * pts * sum(math.log2(s) for s in sizes)
    return dict(bytes=2 * vec, flops=fl)


def _solve_work(spec, nx, nz):
    """Right-hand sides read, solutions written, the operators' nonzeros read and used once."""
    by = fl = 0.0
    for b, (modes, _) in zip(spec.buckets, spec.systems(nx, nz)):
        by += len(modes) * 16.0 * (2 * b["n"] + len(b["indices"]))
        fl += len(modes) * 8.0 * len(b["indices"])
    return dict(bytes=by, flops=fl)


def _step_work(spec, nx, nz, case):
    """The state read and written once a pass and the operators read once a step."""
    stages = {"RK222": 2, "RK443": 4}.get(case["scheme"], 1)
    f, s = _rhs_work(spec, nx, nz), _solve_work(spec, nx, nz)
    return dict(bytes=f["bytes"] + case["steps"] * (s["bytes"] - f["bytes"]),
                flops=case["steps"] * stages * (f["flops"] + s["flops"]))


# ------------------------------------------------------------------------------------------------
# 64-bit results by plain torch: the problem data from its file, dense solves, library transforms

class _Spec:
    """The committed data of a problem."""

    def __init__(self, name, Ra=1e5, nu=0.01 / math.pi):
        z = np.load(os.path.join(PROBLEMS, ("channel_ny129" if name == "channel" else name) + ".npz"))
        meta = json.loads(str(z["meta"]))
        fa, ca = meta["fourier_axes"], meta["cheb_axis"]
        self.lengths = [meta["axes"][a]["L"] for a in fa]
        self.ny, self.ly = (meta["axes"][ca]["N"], meta["axes"][ca]["L"]) if ca >= 0 else (1, 1.0)
        order = lambda o: ([o[a] for a in fa] + [0, 0])[:2] + [o[ca] if ca >= 0 else 0]
        self.factors = [(v, c, order(o)) for v, c, o in meta["factors"]]
        self.outputs = meta["outputs"]
        self.conv = {int(k): z[f"conv_{k}"] for k in meta["lams"]}
        self.b0 = meta["b0"]
        self.buckets = []
        for i, b in enumerate(meta["buckets"]):
            d = {k: z[f"b{i}_{k}"] for k in ("indptr", "indices", "monos", "Mc", "Lc", "col", "row")}
            for p in meta.get("linear_params") or []:
                d["Lc"] = d["Lc"] + {"Ra": Ra, "nu": nu}[p] * z[f"b{i}_dL_{p}"]
            d.update({k: b[k] for k in ("kind", "n", "r", "active", "sign")})
            self.buckets.append(d)

    def systems(self, nx, nz):
        """Per bucket (mode indices, signed wavenumbers) of its systems."""
        out = []
        K = [n // 2 for n in (nx, nz)][: len(self.lengths)]
        for b in self.buckets:
            rng = [np.arange(1, k) if act else np.arange(1) for act, k in zip(b["active"], K)]
            modes = np.stack([g.ravel() for g in np.meshgrid(*rng, indexing="ij")], axis=1) if rng else np.zeros((1, 0), int)
            kw = modes * np.array([2 * np.pi / L for L in self.lengths])
            if len(rng) == 2:
                kw[:, 1] *= b["sign"]
            out.append((modes, kw))
        return out

    def unknowns(self, nx, nz):
        return sum(len(m) * b["n"] for b, (m, _) in zip(self.buckets, self.systems(nx, nz)))

    @staticmethod
    def values(b, kw):
        """Values of M and L of a bucket at wavenumbers kw, (systems, nonzeros) each."""
        mono = np.prod(kw[:, None, :] ** b["monos"][None], axis=2).astype(complex) if kw.shape[1] else \
            np.ones((len(kw), len(b["monos"])), complex)
        return mono @ b["Mc"], mono @ b["Lc"]

    def dense(self, i, vals):
        b = self.buckets[i]
        v = torch.as_tensor(vals, device="cuda")
        A = torch.zeros((len(v), b["n"], b["n"]), dtype=C128, device="cuda")
        rows = np.repeat(np.arange(b["n"]), np.diff(b["indptr"]))
        A[:, torch.as_tensor(rows, device="cuda"), torch.as_tensor(b["indices"].astype(np.int64), device="cuda")] = v
        return A


def _cheb_matrix(m, n):
    """T_k(t_j) on the Gauss nodes t_j = -cos(pi (j + 1/2) / m)."""
    j = torch.arange(m, dtype=torch.float64, device="cuda")[:, None]
    k = torch.arange(n, dtype=torch.float64, device="cuda")[None]
    return torch.cos(math.pi * torch.remainder(k * (2 * j + 1 + 2 * m), 4 * m) / (2 * m))


def _cheb_project(m, n):
    w = 2.0 / m * _cheb_matrix(m, n).T
    w[0] *= 0.5
    return w


def _backward(spec, fields, nx, nz, mx, mz, my):
    """Spectra (fields, Kx, Nz, ny) -> grid values (fields, mx, mz, my), real."""
    g = fields @ _cheb_matrix(my, fields.shape[-1]).T.to(C128) if fields.shape[-1] > 1 else fields
    f, K, nzc, m = g.shape
    if nz:
        h = nz // 2
        full = torch.zeros((f, K, mz, m), dtype=C128, device="cuda")
        full[:, :, :h] = g[:, :, :h]
        full[:, :, mz - h + 1:] = g[:, :, h + 1:]
        g = torch.fft.ifft(full, dim=2) * mz
    if nx:
        full = torch.zeros((f, mx // 2 + 1, g.shape[2], m), dtype=C128, device="cuda")
        full[:, :K] = g
        return torch.fft.irfft(full, n=mx, dim=1) * mx
    return g.real.contiguous()


def _forward(grid, K, nz, ny):
    """Grid values -> kept spectra (fields, K, Nz, ny)."""
    mx, mz, my = grid.shape[1:]
    g = torch.fft.rfft(grid, dim=1)[:, :K] / mx if K > 1 or mx > 1 else grid.to(C128)
    if nz:
        h = nz // 2
        s = torch.fft.fft(g, dim=2) / mz
        g = torch.zeros((g.shape[0], g.shape[1], nz, my), dtype=C128, device="cuda")
        g[:, :, :h] = s[:, :, :h]
        g[:, :, h + 1:] = s[:, :, mz - h + 1:]
    return g @ _cheb_project(my, ny).T.to(C128) if ny > 1 else g


def _exact_rhs(spec, nx, nz, X):
    """F of the state X (per bucket, on the GPU), per bucket."""
    K, nzc, ny = max(nx // 2, 1), max(nz, 1), spec.ny
    mx, mz, my = (3 * nx // 2 or 1), (3 * nz // 2 or 1), (3 * ny // 2 if ny > 1 else 1)
    D = torch.zeros((ny, ny), dtype=torch.float64, device="cuda")     # d/dy on Chebyshev coefficients
    for n in range(ny):
        for k in range(n + 1, ny, 2):
            D[n, k] = 2.0 * k * (0.5 if n == 0 else 1.0) * 2.0 / spec.ly
    systems = spec.systems(nx, nz)
    grids = []
    for v, c, (ox, oz, oy) in spec.factors:
        S = torch.zeros((1, K, nzc, ny), dtype=C128, device="cuda")
        for b, (modes, kw), x in zip(spec.buckets, systems, X):
            at = [(int(n) if ny > 1 else 0, i) for i, (bv, bc, n) in enumerate(b["col"]) if bv == v and bc == c and (n >= 0 or ny == 1)]
            if not at:
                continue
            z = torch.zeros((len(modes), ny), dtype=C128, device="cuda")
            z[:, [n for n, _ in at]] = x[:, [i for _, i in at]]
            w = torch.full((len(modes),), 0.5 ** sum(b["active"]), dtype=C128, device="cuda")
            for axis, o in ((0, ox), (1, oz)):
                if o:
                    w = w * (1j * torch.as_tensor(kw[:, axis], device="cuda")) ** o
            for _ in range(oy):
                z = z @ D.T.to(C128)
            z = z * w[:, None]
            if b["kind"] == "real":
                z = z.real.to(C128)
            jx = torch.as_tensor(modes[:, 0] if nx else np.zeros(len(modes), int), device="cuda")
            jz = torch.as_tensor(modes[:, 1] if nz else np.zeros(len(modes), int), device="cuda")
            slot = jz if b["sign"] > 0 else torch.remainder(-jz, nzc)
            S[0, jx, slot] = z
            mean = (jx == 0) & (jz > 0)
            S[0, jx[mean], torch.remainder(-jz[mean], nzc)] = z[mean].conj()
        grids.append(_backward(spec, S, nx, nz, mx, mz, my)[0])
    H = {}
    for e, c, monos in spec.outputs:
        acc = torch.zeros_like(grids[0])
        for co, fs in monos:
            term = torch.full_like(acc, co[0] if isinstance(co, (list, tuple)) else float(co))
            for f in fs:
                term = term * grids[f]
            acc = acc + term
        H[(e, c)] = _forward(acc[None], K, nz, ny)[0]
    out = []
    for bi, (b, (modes, kw)) in enumerate(zip(spec.buckets, systems)):
        R = torch.zeros((len(modes), b["n"]), dtype=C128, device="cuda")
        jx = torch.as_tensor(modes[:, 0] if nx else np.zeros(len(modes), int), device="cuda")
        jz = torch.as_tensor(modes[:, 1] if nz else np.zeros(len(modes), int), device="cuda")
        slot = jz if b["sign"] > 0 else torch.remainder(-jz, nzc)
        for (e, c), h in H.items():
            at = [(int(n) if ny > 1 else 0, i, int(lam)) for i, (be, bc, n, lam) in enumerate(b["row"]) if be == e and bc == c and (n >= 0 or ny == 1)]
            if not at:
                continue
            lam = max(0, max(l for _, _, l in at))
            z = h[jx, slot] * 2.0 ** sum(b["active"])
            if lam:
                z = z @ torch.as_tensor(spec.conv[lam], device="cuda").T.to(C128)
            if b["kind"] == "real":
                z = z.real.to(C128)
            R[:, [i for _, i, _ in at]] = z[:, [n for n, _, _ in at]]
        for i, mode, pos, v in spec.b0:
            if i == bi:
                hit = np.nonzero(np.all(modes == np.asarray(mode).reshape(1, -1), axis=1))[0]
                if hit.size:
                    R[int(hit[0]), pos] += complex(v[0], v[1])
        out.append(R)
    return out


def _exact_solve(spec, nx, nz, a, b, B):
    """(a M + b L)^-1 B per bucket, dense, some systems at a time."""
    out = []
    for i, (bk, (_, kw), rhs) in enumerate(zip(spec.buckets, spec.systems(nx, nz), B)):
        x = torch.empty_like(rhs)
        for s in range(0, len(kw), 512):
            M, L = spec.values(bk, kw[s:s + 512])
            x[s:s + 512] = torch.linalg.solve(spec.dense(i, a * M + b * L), rhs[s:s + 512].unsqueeze(-1)).squeeze(-1)
        out.append(x)
    return out


def _flat(blocks):
    return torch.cat([x.reshape(-1) for x in blocks])


def _on_gpu(blocks):
    return [torch.as_tensor(np.ascontiguousarray(x, dtype=np.complex128), device="cuda") for x in blocks]


_SBDF = {1: ([1, -1], [1]), 2: ([1.5, -2, 0.5], [2, -1]), 3: ([11 / 6, -3, 1.5, -1 / 3], [3, -3, 1]),
         4: ([25 / 12, -4, 3, -4 / 3, 0.25], [4, -6, 4, -1])}


def _exact_sbdf(spec, nx, nz, X, dt, order, steps):
    """``steps`` SBDF steps from the state X with the lower-order start-up."""
    mats = [spec.values(b, kw) for b, (_, kw) in zip(spec.buckets, spec.systems(nx, nz))]
    Md = [spec.dense(i, m[0]) for i, m in enumerate(mats)]
    Ld = [spec.dense(i, m[1]) for i, m in enumerate(mats)]
    lu = {}
    MX, F = [], []
    for _ in range(steps):
        MX.insert(0, [(M @ x.unsqueeze(-1)).squeeze(-1) for M, x in zip(Md, X)])
        F.insert(0, _exact_rhs(spec, nx, nz, X))
        q = min(order, len(MX))
        a, c = _SBDF[q]
        R = [sum(c[j] * F[j][i] - a[j + 1] / dt * MX[j][i] for j in range(q)) for i in range(len(X))]
        if q not in lu:
            lu[q] = [torch.linalg.lu_factor(a[0] / dt * M + L) for M, L in zip(Md, Ld)]
        X = [torch.linalg.lu_solve(*f, r.unsqueeze(-1)).squeeze(-1) for f, r in zip(lu[q], R)]
    return X


def exact(case, seed):
    kind = case["kind"]
    if kind == "rhs":
        if case["problem"] == "channel" and case["nx"] * case["nz"] > 192 * 192:
            return None
        X = _on_gpu(_smooth(case, seed))
        return _flat(_exact_rhs(_Spec(case["problem"]), case["nx"], case["nz"], X))
    if kind == "solve":
        if case["problem"] == "channel" and case["nx"] * case["nz"] > 64 * 64:
            return None                     # thousands of dense 522 x 522 factorizations
        return _flat(_exact_solve(_Spec(case["problem"]), case["nx"], case["nz"], case["a"], 1.0,
                                  _on_gpu(_rhs_rows(case, seed))))
    if kind == "transforms":
        f, K, nz, ny, mx, mz, my = _transform_sizes(case)
        z, grid = _transform_inputs(case, seed)
        return _backward(None, z, case["nx"], nz, mx, mz, my), _forward(grid, K, nz, ny)
    if kind == "step" and case["problem"] != "channel" and case["scheme"].startswith("SBDF"):
        spec, P = _Spec(case["problem"]), _problem(case)
        X = _on_gpu(_state(case, P, seed))
        return _flat(_exact_sbdf(spec, case["nx"], case["nz"], X, case["dt"], int(case["scheme"][-1]), case["steps"]))
    if kind == "ensemble" and case["scheme"] == "SBDF2" and case["cases"] <= 12:
        _, _, dt, parts = _stack(case, seed)
        out = []
        for nz, ra, states in parts:        # case-major buckets of every resolution, side by side
            done = [_exact_sbdf(_Spec(f"rb_nz{nz}_ra", Ra=float(r)), 4 * nz, 0, _on_gpu(st), dt, 2, case["steps"])
                    for r, st in zip(ra, states)]
            out += [torch.cat(blocks) for blocks in zip(*done)]
        return _flat(out)
    if kind == "core":
        n, _, mats, rhs = _core_mats(case, seed)
        A = np.zeros((case["batch"], n, n), rhs.dtype)
        for k, (_, ip, ix, v) in enumerate(mats):
            A[k, np.repeat(np.arange(n), np.diff(ip)), ix] = v
        A = torch.as_tensor(A, device="cuda")
        A = A.transpose(1, 2) if case["transpose"] else A
        x = torch.linalg.solve(A, torch.as_tensor(rhs, device="cuda").unsqueeze(-1)).squeeze(-1)
        return x.cpu().numpy() if case["where"] == "host" else x
    return None                             # whole 3D steps, Runge-Kutta and large ensembles: minutes
