"""Performance cases of the DG operator path: what a user's program does with this library.

Every case goes through the public Python API (``bosss_b200.operator``,
``bosss_b200.timestepping``) or, where the API is the C header, through the C-ABI call. The
kinds are the configurations that ``bench.py`` and ``bosss_b200/problems.py`` name, at their
sizes and at odd and ragged ones:

* ``transport``: linear upwind transport on a small 2D (or 3D) periodic grid, one residual --
  the smallest call, where launch latency counts;
* ``euler``: compressible Euler / HLLC on a periodic box: residual and adjoint product at the
  same state (``step``: explicit and adjoint codes), or one JVP (Newton-Krylov);
* ``euler_host``: the same pair through the host-buffer entry point, as the C# caller uses it;
* ``rk``: classical Runge-Kutta steps of the Euler operator, one captured graph per step;
* ``sip``: nonlinear diffusion with interior penalty, Dirichlet boundaries: the JVP (the
  operator of matrix-free Newton-GMRES), or residual and adjoint product;
* ``advdiff``: linear advection-diffusion: residual, JVP and VJP;
* ``batch``: many independent advection-diffusion instances of mixed size and degree, tuned
  and captured once, replayed per step;
* ``xdg``: two-phase Poisson with a sphere interface: bulk of both species and interface term;
* ``spmv``: the block-sparse product at the pattern of a DG Jacobian;
* ``newton``: a Newton-GMRES call with a fixed iteration budget (Jacobian assembly, multigrid
  set-up, 30 Krylov iterations per step).
"""
import ctypes
import math

import numpy as np
import torch

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from bosss_b200.timestepping import RungeKutta, RungeKuttaScheme

GAMMA = 1.4
MACH = 1.0 / math.sqrt(GAMMA)
DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # 2D scalar advection, 64x64 quads, k = 2: the smallest configuration of the benchmark
        {"name": "transport2d_64_k2", "kind": "transport", "dim": 2, "n0": 64, "n1": 64, "n2": 1, "k": 2},
        # the headline step: residual + adjoint product, Euler 32^3, k = 3, order 7
        {"name": "euler_32_k3_step", "kind": "euler", "n0": 32, "n1": 32, "n2": 32, "k": 3, "what": "step"},
        # tangent product of the Euler operator on a ragged box (implicit / sensitivity codes)
        {"name": "euler_24x17x13_k2_jvp", "kind": "euler", "n0": 24, "n1": 17, "n2": 13, "k": 2, "what": "jvp"},
        # the headline step from and to host arrays: how the managed caller reaches the library
        {"name": "euler_32_k3_host", "kind": "euler_host", "n0": 32, "n1": 32, "n2": 32, "k": 3},
        # explicit time stepping on a small box: launches and stage updates count
        {"name": "rk4_17x12x9_k2", "kind": "rk", "n0": 17, "n1": 12, "n2": 9, "k": 2, "steps": 3},
        # operator of the matrix-free Newton-GMRES solve, 48^3, k = 2, order 8 (5 nodes)
        {"name": "sip_48_k2_jvp", "kind": "sip", "n0": 48, "n1": 48, "n2": 48, "k": 2, "what": "jvp"},
        # the highest degree of the nonlinear diffusion (9 nodes per direction), ragged grid
        {"name": "sip_21x16x18_k4_step", "kind": "sip", "n0": 21, "n1": 16, "n2": 18, "k": 4, "what": "step"},
        # one linear advection-diffusion instance, all three products, ragged grid
        {"name": "advdiff_20x31x27_k3", "kind": "advdiff", "n0": 20, "n1": 31, "n2": 27, "k": 3},
        # the batched mix: 16 instances of 16^3 .. 32^3 cells, degrees 1 .. 4
        {"name": "batch_16", "kind": "batch", "count": 16, "mix": 5},
        # two-phase Poisson with cut cells
        {"name": "xdg_80_k2", "kind": "xdg", "n": 80, "k": 2},
        # SpMV at the Jacobian's block pattern (k = 2: 10 x 10 blocks, 7 per row), larger than L2
        {"name": "spmv_37x32x33_k2", "kind": "spmv", "n0": 37, "n1": 32, "n2": 33, "k": 2},
        # a whole Newton call with a bounded Krylov budget, multigrid-preconditioned
        {"name": "newton_24_k2", "kind": "newton", "n0": 24, "n1": 24, "n2": 24, "k": 2, "outer": 2, "krylov": 30},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["transport", "euler", "euler", "euler_host", "rk", "sip", "sip", "advdiff", "advdiff",
                       "batch", "xdg", "spmv", "newton"])
    if kind == "transport":
        dim = rng.choice([2, 2, 3])
        if dim == 2:
            return {"kind": kind, "dim": 2, "n0": size(16, 160), "n1": size(16, 160), "n2": 1, "k": rng.randint(1, 4)}
        return {"kind": kind, "dim": 3, "n0": size(8, 40), "n1": size(8, 40), "n2": size(8, 40), "k": rng.randint(1, 4)}
    if kind in ("euler", "euler_host"):
        k = rng.randint(1, 4)
        top = {1: 40, 2: 36, 3: 32, 4: 26}[k]
        c = {"kind": kind, "n0": size(6, top), "n1": size(6, top), "n2": size(6, top), "k": k}
        if kind == "euler":
            c["what"] = rng.choice(["step", "jvp"])
        return c
    if kind == "rk":
        return {"kind": kind, "n0": size(6, 24), "n1": size(6, 24), "n2": size(6, 24), "k": rng.randint(1, 3),
                "steps": rng.randint(1, 4)}
    if kind == "sip":
        k = rng.randint(1, 4)
        top = {1: 56, 2: 48, 3: 32, 4: 22}[k]
        return {"kind": kind, "n0": size(6, top), "n1": size(6, top), "n2": size(6, top), "k": k,
                "what": rng.choice(["step", "jvp"])}
    if kind == "advdiff":
        return {"kind": kind, "n0": size(8, 48), "n1": size(8, 48), "n2": size(8, 48), "k": rng.randint(1, 4)}
    if kind == "batch":
        return {"kind": kind, "count": size(3, 20), "mix": rng.randint(1, 100000)}
    if kind == "xdg":
        return {"kind": kind, "n": size(20, 84), "k": rng.choice([1, 2, 2])}
    if kind == "spmv":
        k = rng.randint(1, 4)
        top = {1: 44, 2: 36, 3: 26, 4: 20}[k]
        return {"kind": kind, "n0": size(8, top), "n1": size(8, top), "n2": size(8, top), "k": k}
    return {"kind": "newton", "n0": size(8, 24), "n1": size(8, 24), "n2": size(8, 24), "k": rng.randint(1, 2),
            "outer": 2, "krylov": rng.randint(15, 30)}


# ------------------------------------------------------------------------------------ inputs
def gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def uniform(g, *shape):
    return torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g) * 2 - 1


def modes(dim, k):
    """Exponents of the total-degree basis in the library's polynomial order."""
    m = []
    for deg in range(k + 1):
        if dim == 2:
            m += [(a, deg - a) for a in range(deg + 1)]
        else:
            m += [(a, b, deg - a - b) for a in range(deg + 1) for b in range(deg - a + 1)]
    return m


def np_of(dim, k):
    return len(modes(dim, k))


def legendre(k, x):
    """Normalised Legendre polynomials and derivatives at x: two arrays [len(x), k + 1]."""
    x = np.asarray(x, dtype=np.float64)
    L, D = np.empty((len(x), k + 1)), np.empty((len(x), k + 1))
    for a in range(k + 1):
        c = np.zeros(a + 1)
        c[a] = math.sqrt((2 * a + 1) / 2.0)
        L[:, a] = np.polynomial.legendre.legval(x, c)
        D[:, a] = np.polynomial.legendre.legval(x, np.polynomial.legendre.legder(c)) if a else 0.0
    return L, D


def tables(dim, k, pts):
    """Basis values and reference gradients at the tensor points pts (one 1D array per
    direction): phi[q, n], dphi[d][q, n], coordinates [q, dim]."""
    idx = np.meshgrid(*[np.arange(len(p)) for p in pts], indexing="ij")
    one = [legendre(k, p) for p in pts]
    phi, dphi = [], [[] for _ in range(dim)]
    for e in modes(dim, k):
        v = [one[d][0][idx[d].ravel(), e[d]] for d in range(dim)]
        w = [one[d][1][idx[d].ravel(), e[d]] for d in range(dim)]
        phi.append(np.prod(v, axis=0))
        for d in range(dim):
            dphi[d].append(np.prod([w[i] if i == d else v[i] for i in range(dim)], axis=0))
    x = np.stack([pts[d][idx[d].ravel()] for d in range(dim)], axis=1)

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    return t(np.stack(phi, 1)), [t(np.stack(d, 1)) for d in dphi], t(x)


def project(dim, k, nq, h, nodal):
    """L2 projection of nodal values [..., nq^dim] (iid at the Gauss nodes) onto the basis."""
    x, w = np.polynomial.legendre.leggauss(nq)
    phi, _, _ = tables(dim, k, [x] * dim)
    W = torch.from_numpy(np.prod(np.meshgrid(*[w] * dim, indexing="ij"), axis=0).ravel()).to(DEV)
    return (nodal * W) @ phi * math.sqrt(math.prod(0.5 * v for v in h))


def box(case):
    """Cells per direction and cell widths: the cells of the unit box cut 1/n0 wide (cubic cells
    for Euler, the unit cube for the scalar problems)."""
    n = [case["n0"], case["n1"], case["n2"]][: case.get("dim", 3)]
    if case["kind"] in ("euler", "euler_host", "rk"):
        return n, [1.0 / n[0]] * len(n)
    return n, [1.0 / v for v in n]


def euler_state(g, n, k, h):
    """rho = 1 + 0.1 U, u_d = 0.3 U, p = 1 + 0.1 U at the volume nodes, projected: [cells, 5, Np]."""
    J, nq = math.prod(n), k + 1
    rho = 1.0 + 0.1 * uniform(g, J, nq ** 3)
    vel = 0.3 * uniform(g, 3, J, nq ** 3)
    p = 1.0 + 0.1 * uniform(g, J, nq ** 3)
    E = p / (GAMMA - 1.0) + 0.5 * GAMMA * MACH ** 2 * rho * (vel ** 2).sum(0)
    f = torch.stack([rho, rho * vel[0], rho * vel[1], rho * vel[2], E], 1)
    return project(3, k, nq, h, f)


def inputs(case, seed):
    """The vectors of a case, from the seed alone (torch tensors, flat)."""
    g, kind = gen(seed), case["kind"]
    if kind in ("transport", "euler", "euler_host", "rk", "sip", "advdiff", "newton"):
        n, h = box(case)
        J, k, dim = math.prod(n), case["k"], len(n)
        Np = np_of(dim, k)
        if kind in ("euler", "euler_host", "rk"):
            U = euler_state(g, n, k, h).reshape(-1)
        elif kind == "sip":
            U = project(3, k, k + 1, h, uniform(g, J, (k + 1) ** 3)).reshape(-1)
        elif kind == "newton":
            U = 0.1 * project(3, k, k + 1, h, uniform(g, J, (k + 1) ** 3)).reshape(-1)
        else:
            U = uniform(g, J * Np)
        return {"U": U.contiguous(), "V": uniform(g, U.numel()), "W": uniform(g, U.numel()),
                "vel": [float(v) for v in uniform(g, 3).cpu()]}
    if kind == "batch":
        insts = batch_mix(case)
        J = [i["n"] ** 3 * np_of(3, i["k"]) for i in insts]
        return {"U": uniform(g, sum(J)), "W": uniform(g, sum(J)), "vel": uniform(g, len(J), 3).cpu().tolist()}
    if kind == "xdg":
        N = case["n"] ** 3 * np_of(3, case["k"])
        return {"UA": uniform(g, N), "UB": uniform(g, N), "center": [0.05 * float(v) for v in uniform(g, 3).cpu()]}
    rp, ci = pattern([case["n0"], case["n1"], case["n2"]])
    b = np_of(3, case["k"])
    return {"rp": rp, "ci": ci, "vals": uniform(g, len(ci), b, b), "x": uniform(g, (len(rp) - 1) * b)}


def batch_mix(case):
    r = np.random.default_rng(case["mix"])
    return [{"n": int(r.choice([16, 24, 32])), "k": int(r.integers(1, 5))} for _ in range(case["count"])]


def pattern(n):
    """Block rows of a hex grid (generator order): the cell and its face neighbours, sorted."""
    J = math.prod(n)
    idx = np.arange(J).reshape(n)
    cols, ok = [idx.ravel()], [np.ones(J, bool)]
    for d in range(3):
        for s in (-1, 1):
            c = np.roll(idx, -s, axis=d)
            v = np.ones(n, bool)
            cut = [slice(None)] * 3
            cut[d] = 0 if s < 0 else n[d] - 1
            v[tuple(cut)] = False
            cols.append(c.ravel())
            ok.append(v.ravel())
    cm, om = np.stack(cols, 1), np.stack(ok, 1)
    key = np.where(om, cm, J + 1)
    order = np.argsort(key, axis=1, kind="stable")
    cm, om = np.take_along_axis(cm, order, 1), np.take_along_axis(om, order, 1)
    rp = np.zeros(J + 1, np.int64)
    rp[1:] = np.cumsum(om.sum(1))
    return rp, cm[om].astype(np.int32)


# ------------------------------------------------------------------------------------ operators
def scalar_operator(n, h, k, periodic, comps, quad, lo=0.0):
    nodes = [np.linspace(lo, lo + v * w, v + 1) for v, w in zip(n, h)]
    grid = (O.Cartesian2DGrid if len(n) == 2 else O.Cartesian3DGrid)(*nodes, *[periodic] * len(n))
    op = O.DifferentialOperator(["u"], [], ["R"], quad)
    for c in comps:
        op.EquationComponents["R"].Add(c)
    op.Commit()
    return op, [O.DGField(grid, k, "u")], [O.DGField(grid, k, "R")]


def euler_evaluator(n, h, k):
    grid = O.Cartesian3DGrid(*[np.linspace(0.0, v * w, v + 1) for v, w in zip(n, h)], True, True, True)
    names = ["rho", "m0", "m1", "m2", "rhoE"]
    op = O.DifferentialOperator(names, [], ["R_" + s for s in names], O.QuadOrderFunc.FixedOrder(2 * k + 1))
    mat = O.Material(GAMMA)
    op.EquationComponents["R_rho"].Add(O.OptimizedHLLCDensityFlux(mat, 3))
    for d in range(3):
        op.EquationComponents["R_m%d" % d].Add(O.OptimizedHLLCMomentumFlux(mat, d, 3))
    op.EquationComponents["R_rhoE"].Add(O.OptimizedHLLCEnergyFlux(mat, 3))
    op.Commit()
    return op.GetEvaluatorEx([O.DGField(grid, k, s) for s in names], None, [O.DGField(grid, k, "R_" + s) for s in names])


class Instance:
    """One instance of a batch: its operator and grid descriptors."""

    def __init__(self, op, dom, cod):
        self.op, self.dom, self.cod = op, dom, cod

    def descs(self):
        return (self.op.descriptor([f.degree for f in self.dom], [f.degree for f in self.cod], 3),
                self.dom[0].grid.desc())


def advdiff_operator(n, h, k, vel):
    return scalar_operator(n, h, k, True, [O.ScalarTransportFlux(vel, "u"), O.SIPLaplace(4.0, "u", nu0=0.01)],
                           O.QuadOrderFunc.Linear())


def sip_operator(n, h, k, source=0.0):
    comps = [O.SIPLaplace(4.0, "u", nu0=1.0, nu2=1.0)] + ([O.ConstantSource(source, "u")] if source else [])
    return scalar_operator(n, h, k, False, comps, O.QuadOrderFunc.NonLinear(3))


# ------------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind, x = case["kind"], inputs(case, seed)
    s = {"case": case, "x": x}
    if kind in ("transport", "euler", "euler_host", "rk", "sip", "advdiff", "newton"):
        n, h = box(case)
        k = case["k"]
        if kind == "transport":
            op, dom, cod = scalar_operator(n, h, k, True, [O.ScalarTransportFlux(x["vel"][: len(n)], "u")],
                                           O.QuadOrderFunc.FixedOrder(2 * k + 1))
            s["ev"] = op.GetEvaluatorEx(dom, None, cod)
        elif kind in ("sip", "newton"):
            op, dom, cod = sip_operator(n, h, k, 1.0 if kind == "newton" else 0.0)
            s["ev"] = op.GetEvaluatorEx(dom, None, cod)
        elif kind == "advdiff":
            op, dom, cod = advdiff_operator(n, h, k, x["vel"])
            s["ev"] = op.GetEvaluatorEx(dom, None, cod)
        else:
            s["ev"] = euler_evaluator(n, h, k)
        if kind == "rk":
            s["rk"] = RungeKutta(RungeKuttaScheme.RungeKutta1901(), s["ev"])
            s["u"] = x["U"].clone()
        elif kind == "euler_host":
            for v in ("U", "W"):
                s[v] = x[v].cpu().pin_memory().numpy()
            s["R"] = torch.zeros(len(s["U"]), dtype=torch.float64).pin_memory().numpy()
            s["G"] = torch.zeros(len(s["U"]), dtype=torch.float64).pin_memory().numpy()
        elif kind == "newton":
            s["U"] = x["U"].cpu().numpy()
        else:
            s["R"], s["G"], s["JV"] = (torch.zeros_like(x["U"]) for _ in range(3))
    elif kind == "batch":
        insts = []
        for i, vel in zip(batch_mix(case), x["vel"]):
            insts.append(Instance(*advdiff_operator([i["n"]] * 3, [1.0 / i["n"]] * 3, i["k"], vel)))
        s["B"] = O.BatchEvaluator(insts)
        s["R"], s["G"] = torch.zeros_like(x["U"]), torch.zeros_like(x["U"])
        torch.cuda.synchronize()
        s["B"].autotune(x["U"], x["W"], s["R"], s["G"])
        s["B"].capture(x["U"], x["W"], s["R"], s["G"])
    elif kind == "xdg":
        n, k, ops = case["n"], case["k"], []
        for mu in (1.0, 10.0):
            op, dom, _ = scalar_operator([n] * 3, [2.0 / n] * 3, k, False,
                                         [O.SIPLaplace(4.0, "u", nu0=mu), O.ConstantSource(1.0, "u")],
                                         O.QuadOrderFunc.FixedOrder(5), lo=-1.0)
            ops.append(op)
        s["X"] = O.XdgEvaluator(ops[0], ops[1], dom[0].grid, k, x["center"], 0.4)
        s["X"].SetInterface(1.0, 10.0, 4.0)
        s["RA"], s["RB"] = torch.zeros_like(x["UA"]), torch.zeros_like(x["UB"])
    else:
        J = len(x["rp"]) - 1
        s["A"] = O.BlockMsrMatrix.from_blocks(J, J, x["rp"], x["ci"], x["vals"].cpu().numpy())
        s["y"] = torch.zeros_like(x["x"])
        del x["vals"]
    torch.cuda.synchronize()
    return s


def run(s):
    case, x = s["case"], s["x"]
    kind = case["kind"]
    if kind == "transport":
        return s["ev"].Evaluate(1.0, 0.0, s["R"], x["U"])
    if kind in ("euler", "sip"):
        if case["what"] == "jvp":
            return s["ev"].jvp(x["U"], x["V"], s["JV"])
        return s["ev"].Evaluate(1.0, 0.0, s["R"], x["U"]), s["ev"].vjp(x["U"], x["W"], s["G"])
    if kind == "euler_host":
        return s["ev"].residual_vjp(s["U"], s["W"], s["R"], s["G"])
    if kind == "rk":
        s["u"].copy_(x["U"])
        return s["rk"].PerformDevice(s["u"], time_step(case), case["steps"])
    if kind == "advdiff":
        return (s["ev"].Evaluate(1.0, 0.0, s["R"], x["U"]), s["ev"].jvp(x["U"], x["V"], s["JV"]),
                s["ev"].vjp(x["U"], x["W"], s["G"]))
    if kind == "batch":
        s["B"].replay()
        return s["R"], s["G"]
    if kind == "xdg":
        s["X"].Evaluate(0, 1.0, 0.0, s["RA"], x["UA"])
        s["X"].Evaluate(1, 1.0, 0.0, s["RB"], x["UB"])
        s["X"].EvaluateInterface(1.0, x["UA"], x["UB"], s["RA"], s["RB"])
        return s["RA"], s["RB"]
    if kind == "spmv":
        st = torch.cuda.current_stream().cuda_stream
        C.check(C.lib().bosss_b200_bsr_spmv_device(s["A"].handle, 1.0, C.ptr(x["x"]), 0.0, C.ptr(s["y"]),
                                                   ctypes.c_void_p(st if st else C.CUDA_STREAM_LEGACY)))
        return s["y"]
    U, _ = s["ev"].NewtonSolve(s["U"], rtol=1e-14, max_outer=case["outer"], restart=case["krylov"],
                               max_krylov=case["krylov"], inner_rtol=1e-14, precond=2)
    return U


def time_step(case):
    """An explicit step: a twentieth of a cell width over (2 k + 1), sound speed near 1."""
    return 0.05 / case["n0"] / (2 * case["k"] + 1)


# ------------------------------------------------------------------------------------ work
def tensor_flops(k, q, grad):
    """Flops of one field's interpolation or projection at q^3 volume nodes by sum
    factorisation, and of its traces on six faces (own side)."""
    pairs = (k + 1) * (k + 2) // 2
    vol = 2 * (np_of(3, k) * q + pairs * q * q + (k + 1) * q ** 3) * (4 if grad else 1)
    face = 6 * 2 * (np_of(3, k) + pairs * q + (k + 1) * q * q) * (2 if grad else 1)
    return vol + face


def work(case):
    kind = case["kind"]
    if kind in ("transport", "euler", "euler_host", "rk", "sip", "advdiff", "newton"):
        n, _ = box(case)
        J, k, dim = math.prod(n), case["k"], len(n)
        nv = 5 if kind in ("euler", "euler_host", "rk") else 1
        N = J * nv * np_of(dim, k)
        # a linear constant-coefficient form is a stencil of 1D products in the modes
        lin = J * np_of(dim, k) * 2 * dim * 6
        eul = J * 5 * 3 * tensor_flops(k, k + 1, False) + J * ((k + 1) ** 3 * 60 + 3 * (k + 1) ** 2 * 150)
        sip = J * 2 * tensor_flops(k, 2 * k + 1, True) + J * (2 * k + 1) ** 3 * 20
        if kind == "transport":
            return {"bytes": 16 * N, "flops": lin}
        if kind == "advdiff":
            return {"bytes": (16 + 24 + 24) * N, "flops": 3 * lin}
        if kind in ("euler", "sip"):
            f = eul if kind == "euler" else sip
            return {"bytes": 24 * N, "flops": 2 * f} if case["what"] == "jvp" else {"bytes": (16 + 24) * N, "flops": 3 * f}
        if kind == "euler_host":
            return {"bytes": 32 * N, "flops": 3 * eul}
        if kind == "rk":
            return {"bytes": case["steps"] * 4 * 32 * N, "flops": case["steps"] * 4 * eul}
        steps, its = case["outer"], case["krylov"]
        blocks = 7 * J * np_of(3, k) ** 2 * 8
        return {"bytes": steps * its * (2 * blocks + (24 + 8 * its) * N), "flops": steps * its * 2 * sip}
    if kind == "batch":
        N = sum(i["n"] ** 3 * np_of(3, i["k"]) for i in batch_mix(case))
        return {"bytes": 40 * N, "flops": 2 * N * 36}
    if kind == "xdg":
        N = case["n"] ** 3 * np_of(3, case["k"])
        return {"bytes": 32 * N, "flops": 2 * N * 36}
    J, b = case["n0"] * case["n1"] * case["n2"], np_of(3, case["k"])
    nnz = 7 * J - 2 * (case["n1"] * case["n2"] + case["n0"] * case["n2"] + case["n0"] * case["n1"])
    return {"bytes": nnz * (b * b * 8 + 4) + 8 * J + 16 * J * b, "flops": 2 * nnz * b * b}


# ------------------------------------------------------------------------------------ the results in 64 bits
class Dense:
    """A DG operator by dense tables, face by face, in differentiable torch (64 bits):
    ``volume(U, G) -> (fV, fG)`` and ``face(UA, GA, UB, GB, d, pnlty) -> (gA, GA, gB, GB)``
    give the coefficients of the test functions and of their gradients; ``bound`` the terms of
    the faces of a non-periodic box (own side, outward normal ``sign`` along d)."""

    def __init__(self, n, h, k, nq, nv, periodic, grad, volume, face, bound=None, pen=0.0):
        self.n, self.h, self.nv, self.periodic, self.grad, self.pen = n, h, nv, periodic, grad, pen
        self.volume, self.face, self.bound = volume, face, bound
        dim = self.dim = len(n)
        x, w = np.polynomial.legendre.leggauss(nq)

        def ws(m):
            return torch.from_numpy(np.prod(np.meshgrid(*[w] * m, indexing="ij"), axis=0).ravel()).to(DEV)
        detJ = math.prod(0.5 * v for v in h)
        self.sc = 1.0 / math.sqrt(detJ)
        self.two = [2.0 / v for v in h]
        self.Np = np_of(dim, k)
        self.vt = tables(dim, k, [x] * dim)[:2]
        self.vw = ws(dim) * detJ * self.sc
        self.ft, self.fw = {}, []
        for d in range(dim):
            self.fw.append(ws(dim - 1) * (detJ / (0.5 * h[d])) * self.sc)
            for s in (0, 1):
                pts = [np.array([2.0 * s - 1.0]) if i == d else x for i in range(dim)]
                self.ft[d, s] = tables(dim, k, pts)[:2]
        # 1 / cell length scale: half the surface (boundary faces twice) over the volume
        cj = torch.zeros(n, dtype=torch.float64, device=DEV)
        for d in range(dim):
            c = torch.full((n[d],), 2.0, dtype=torch.float64, device=DEV)
            if not periodic:
                c[0] += 1
                c[-1] += 1
            cj = cj + (c / h[d]).reshape([-1 if i == d else 1 for i in range(dim)])
        self.cj = 0.5 * cj

    def at(self, U, t):
        phi, dphi = t
        v = self.sc * (U @ phi.T)
        g = [self.sc * self.two[d] * (U @ dphi[d].T) for d in range(self.dim)] if self.grad else None
        return v, g

    def test(self, fV, fG, t, w):
        phi, dphi = t
        r = 0
        if fV is not None:
            r = r + (fV * w) @ phi
        if fG is not None:
            for d in range(self.dim):
                if fG[d] is not None:
                    r = r + self.two[d] * ((fG[d] * w) @ dphi[d])
        return r

    def __call__(self, flat):
        dim, n = self.dim, self.n
        U = flat.reshape(*n, self.nv, self.Np)
        v, g = self.at(U, self.vt)
        R = self.test(*self.volume(v, g), self.vt, self.vw)
        for d in range(dim):
            if self.periodic:
                A, B = U, torch.roll(U, -1, d)
                cA, cB = self.cj, torch.roll(self.cj, -1, d)
            else:
                A, B = U.narrow(d, 0, n[d] - 1), U.narrow(d, 1, n[d] - 1)
                cA, cB = self.cj.narrow(d, 0, n[d] - 1), self.cj.narrow(d, 1, n[d] - 1)
            tA, tB = self.ft[d, 1], self.ft[d, 0]
            p = (self.pen * torch.maximum(cA, cB))[..., None, None]
            (vA, gA), (vB, gB) = self.at(A, tA), self.at(B, tB)
            fA, FA, fB, FB = self.face(vA, gA, vB, gB, d, p)
            rA, rB = self.test(fA, FA, tA, self.fw[d]), self.test(fB, FB, tB, self.fw[d])
            if self.periodic:
                R = R + rA + torch.roll(rB, 1, d)
                continue
            z = torch.zeros_like(U.narrow(d, 0, 1))
            R = R + torch.cat([rA, z], d) + torch.cat([z, rB], d)
            for s in (0, 1):
                t, at = self.ft[d, s], 0 if s == 0 else n[d] - 1
                p = (2.0 * self.pen * self.cj.narrow(d, at, 1))[..., None, None]
                vI, gI = self.at(U.narrow(d, at, 1), t)
                r = self.test(*self.bound(vI, gI, d, 2.0 * s - 1.0, p), t, self.fw[d])
                z = torch.zeros([n[i] if i != d else n[d] - 1 for i in range(dim)] + [self.nv, self.Np],
                                dtype=torch.float64, device=DEV)
                R = R + (torch.cat([r, z], d) if s == 0 else torch.cat([z, r], d))
        return R.reshape(-1)

    def residual(self, U):
        with torch.no_grad():
            return self(U)

    def vjp(self, U, W):
        u = U.clone().requires_grad_(True)
        return torch.autograd.grad(self(u), u, W)[0]

    def jvp(self, U, V):
        return torch.func.jvp(self, (U,), (V,))[1]


def dense_scalar(n, h, k, nq, periodic, vel=None, nu=None, nu2=0.0, source=0.0):
    """Upwind transport + interior penalty diffusion nu + nu2 u^2 (penalty base 4) + source."""
    dim = len(n)
    pen = 4.0 * max((k + 1.0) * (k + dim) / dim, (k + 1.0) ** 2)

    def visc(u):
        return nu + nu2 * u * u

    def volume(u, g):
        fG = [torch.zeros_like(u) for _ in range(dim)]
        for d in range(dim):
            if vel is not None:
                fG[d] = fG[d] - vel[d] * u
            if nu is not None:
                fG[d] = fG[d] - visc(u) * g[d]
        return (torch.full_like(u, source) if source else None), fG

    def face(a, ga, b, gb, d, p):
        f, SA, SB = 0.0, None, None
        if vel is not None:
            f = f + vel[d] * (a if vel[d] > 0 else b)
        if nu is not None:
            na, nb = visc(a), visc(b)
            f = f + 0.5 * (na * ga[d] + nb * gb[d]) - p * (a - b) * torch.where(na.abs() > nb.abs(), na, nb)
            SA = [0.5 * na * (a - b) if i == d else None for i in range(dim)]
            SB = [0.5 * nb * (a - b) if i == d else None for i in range(dim)]
        return f, SA, -f, SB

    def bound(a, ga, d, sign, p):   # homogeneous Dirichlet
        na = visc(a)
        return na * ga[d] * sign - na * a * p, [na * a * sign if i == d else None for i in range(dim)]

    return Dense(n, h, k, nq, 1, periodic, nu is not None, volume, face, bound, pen)


def dense_euler(n, h, k):
    """Compressible Euler with the HLLC flux (pressure scaled by 1 / (gamma Ma^2))."""
    MS = GAMMA * MACH * MACH

    def parts(U):
        r, m, E = U[..., 0, :], [U[..., 1 + d, :] for d in range(3)], U[..., 4, :]
        u = [v / r for v in m]
        p = (E - 0.5 * MS * sum(a * b for a, b in zip(m, u))) * (GAMMA - 1.0)
        return r, m, E, u, p

    def volume(U, _):
        r, m, E, u, p = parts(U)
        fG = []
        for d in range(3):
            rows = [m[d]] + [m[c] * u[d] + (p / MS if c == d else 0.0) for c in range(3)] + [u[d] * (E + p)]
            fG.append(-torch.stack(rows, -2))
        return None, fG

    def face(A, _, B, __, d, ___):
        rA, mA, EA, uA, pA = parts(A)
        rB, mB, EB, uB, pB = parts(B)
        unA, unB = uA[d], uB[d]
        cA, cB = torch.sqrt(pA / rA) / MACH, torch.sqrt(pB / rB) / MACH
        pS = 0.5 * (pA + pB) - (unB - unA) * 0.25 * (cA + cB) * (rA + rB) * 0.5 * MS
        pS = torch.clamp(pS, min=0.0)
        G2 = 0.5 * (GAMMA + 1.0) / GAMMA
        one = torch.ones_like(pS)
        qA = torch.sqrt(torch.where(pS > pA, 1.0 + G2 * (pS / pA - 1.0), one))
        qB = torch.sqrt(torch.where(pS > pB, 1.0 + G2 * (pS / pB - 1.0), one))
        sA, sB = unA - cA * qA, unB + cB * qB
        kA, kB = rA * (sA - unA), rB * (sB - unB)
        S = (kB * unB - kA * unA + (pA - pB) / MS) / (kB - kA)
        left = S > 0.0

        def pick(a, b):
            return torch.where(left, a, b)
        r, E, p, un, s = pick(rA, rB), pick(EA, EB), pick(pA, pB), pick(unA, unB), pick(sA, sB)
        m = [pick(a, b) for a, b in zip(mA, mB)]
        star = torch.where(left, s <= 0.0, s >= 0.0)
        ratio = (s - un) / (s - S)
        f = [un * r] + [un * m[c] + (p / MS if c == d else 0.0) for c in range(3)] + [un * (E + p)]
        mod = [r * ratio] + [r * ratio * (S if c == d else m[c] / r) for c in range(3)]
        mod += [ratio * (E + (r * S * MS + p / (s - un)) * (S - un))]
        own = [r] + m + [E]
        f = torch.stack([torch.where(star, a + s * (b - c), a) for a, b, c in zip(f, mod, own)], -2)
        return f, None, -f, None

    return Dense(n, h, k, k + 1, 5, True, False, volume, face)


def exact(case, seed):
    kind, x = case["kind"], inputs(case, seed)
    if kind in ("xdg", "newton"):
        return None   # cut-cell rules and truncated Krylov iterations have no plain restatement
    if kind == "spmv":
        J, b = len(x["rp"]) - 1, x["vals"].shape[-1]
        ci = torch.from_numpy(x["ci"].astype(np.int64)).to(DEV)
        rows = torch.from_numpy(np.repeat(np.arange(J), np.diff(x["rp"]))).to(DEV)
        prod = torch.einsum("nij,nj->ni", x["vals"], x["x"].reshape(J, b)[ci])
        return torch.zeros(J, b, dtype=torch.float64, device=DEV).index_add_(0, rows, prod).reshape(-1)
    if kind == "batch":
        R, G, at = [], [], 0
        for i, vel in zip(batch_mix(case), x["vel"]):
            N = i["n"] ** 3 * np_of(3, i["k"])
            D = dense_scalar([i["n"]] * 3, [1.0 / i["n"]] * 3, i["k"], i["k"] + 1, True, vel, 0.01)
            R.append(D.residual(x["U"][at:at + N]))
            G.append(D.vjp(x["U"][at:at + N], x["W"][at:at + N]))
            at += N
        return torch.cat(R), torch.cat(G)
    n, h = box(case)
    k = case["k"]
    if kind == "transport":
        return dense_scalar(n, h, k, k + 1, True, x["vel"]).residual(x["U"])
    if kind == "advdiff":
        D = dense_scalar(n, h, k, k + 1, True, x["vel"], 0.01)
        return D.residual(x["U"]), D.jvp(x["U"], x["V"]), D.vjp(x["U"], x["W"])
    D = dense_scalar(n, h, k, 2 * k + 1, False, None, 1.0, 1.0) if kind == "sip" else dense_euler(n, h, k)
    if kind == "rk":
        a = [[0, 0, 0, 0], [0.5, 0, 0, 0], [0, 0.5, 0, 0], [0, 0, 1, 0]]
        b = [1 / 6, 2 / 6, 2 / 6, 1 / 6]
        u, dt = x["U"], time_step(case)
        for _ in range(case["steps"]):
            ks = []
            for s in range(4):
                ks.append(D.residual(u - dt * sum((a[s][r] * ks[r] for r in range(s)), torch.zeros_like(u))))
            u = u - dt * sum(b[s] * ks[s] for s in range(4))
        return u
    if case.get("what") == "jvp":
        return D.jvp(x["U"], x["V"])
    return D.residual(x["U"]), D.vjp(x["U"], x["W"])
