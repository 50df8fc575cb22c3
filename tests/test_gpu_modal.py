"""Linear constant-coefficient scalar operators on the modal kernel: residual, JVP and VJP against
the oracle and the quadrature kernels at the sizes where tiles are cut (one cell, two periodic
cells, sizes around the tile extents), in both cell orders, with every boundary kind, on cell
ranges and on vectors that start at an odd double."""
import ctypes

import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the parity bar of every FP64 kernel against the oracle


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def make(n, k, comps, periodic, order=C.CELLS_GENERATOR, quad=None):
    nodes = [np.linspace(0.1 * d, 0.1 * d + 1.0 + 0.3 * d, v + 1) for d, v in enumerate(n)]
    g = (O.Cartesian2DGrid if len(n) == 2 else O.Cartesian3DGrid)(*nodes, *periodic, cell_order=order)
    op = O.DifferentialOperator(["u"], [], ["R"], quad or O.QuadOrderFunc.Linear())
    for c in comps:
        op.EquationComponents["R"].Add(c)
    op.Commit()
    return op, g, [O.DGField(g, k, "u")], [O.DGField(g, k, "R")]


def comps_of(kind, dim):
    vel = [0.7, -0.4, 0.3][:dim]
    sip = O.SIPLaplace(4.0, "u", nu0=0.3, g0=0.2, g1=(0.5, -0.3, 0.1), g2=(0.4, 0.2, -0.6))
    if kind == "transport":
        return [O.ScalarTransportFlux(vel, "u")]
    if kind == "neumann":
        return [O.ScalarTransportFlux([-v for v in vel], "u"), O.SIPLaplace(4.0, "u", nu0=-0.2, dirichlet=False)]
    return [O.ScalarTransportFlux(vel, "u"), sip, O.ConstantSource(1.3, "u")]


CASES = [((1, 1, 1), (True, True, True)), ((2, 1, 3), (True, True, True)), ((5, 4, 9), (False, False, False)),
         ((9, 5, 8), (True, False, True)), ((3, 17, 2), (False, True, False)),
         ((1, 1), (True, True)), ((7, 33), (False, False)), ((18, 3), (True, False))]


@pytest.mark.parametrize("kind", ["transport", "dirichlet", "neumann"])
@pytest.mark.parametrize("n,periodic", CASES, ids=lambda v: "x".join(str(int(i)) for i in v))
def test_modal_matches_oracle(n, periodic, kind):
    import torch
    dim = len(n)
    for k in range(0 if kind == "transport" else 1, 5):
        for order in ([C.CELLS_GENERATOR, C.CELLS_GLOBALID] if dim == 3 and k in (1, 4) else [C.CELLS_GENERATOR]):
            op, g, dom, cod = make(n, k, comps_of(kind, dim), periodic, order)
            desc = (op.descriptor([k], [k], dim), g.desc())
            r = np.random.default_rng(k)
            U, V, prev = (r.uniform(-1, 1, g.NoOfCells * dom[0].Np) for _ in range(3))
            pad = torch.zeros(2 * U.size + 1, dtype=torch.float64, device="cuda")
            u, out = pad[1:U.size + 1], pad[U.size + 1:]     # u starts at an odd double
            u.copy_(torch.from_numpy(U))
            v = torch.from_numpy(V).cuda()
            out.copy_(torch.from_numpy(prev))
            with op.GetEvaluatorEx(dom, None, cod) as ev:
                assert [ev.kernel_info(m)[0] for m in range(3)] == [5, 5, 5]
                ev.Evaluate(0.7, 0.3, out, u)
                ref = 0.3 * prev + 0.7 * orc.evaluate(*desc, U)
                assert rel(out.cpu().numpy(), ref) <= TOL, (k, order)
                assert rel(ev.jvp(u, v).cpu().numpy(), orc.jvp(*desc, U, V)) <= TOL, (k, order)
                assert rel(ev.vjp(u, v).cpu().numpy(), orc.vjp(*desc, U, V)) <= TOL, (k, order)


@pytest.mark.parametrize("quad", [O.QuadOrderFunc.NonLinear(2), O.QuadOrderFunc.NonLinear(3)], ids=["nl2", "nl3"])
def test_modal_matches_higher_rules_and_ranges(quad):
    """Rules above the exact one give the same integrals; a cell range writes its cells only."""
    import torch
    n, k = (6, 5, 7), 2
    op, g, dom, cod = make(n, k, comps_of("dirichlet", 3), (False, True, False), quad=quad)
    N, Np = g.NoOfCells * dom[0].Np, dom[0].Np
    U = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, N)).cuda()
    with op.GetEvaluatorEx(dom, None, cod) as ev, op.GetEvaluatorEx(dom, None, cod, kernel=C.KERNEL_GENERIC) as eg:
        a, b = torch.zeros_like(U), torch.zeros_like(U)
        ev.Evaluate(1.0, 0.0, a, U)
        eg.Evaluate(1.0, 0.0, b, U)
        torch.cuda.synchronize()
        assert rel(a.cpu().numpy(), b.cpu().numpy()) <= TOL
        for lo, hi in ((0, 1), (34, 36), (13, 171), (0, g.NoOfCells)):
            c = torch.full_like(U, 9.0)
            C.check(C.lib().bosss_b200_apply_device(ev.handle, 0, 1.0, 0.0, C.ptr(U), None, C.ptr(c), 0.0, lo, hi,
                                                    ctypes.c_void_p(C.CUDA_STREAM_LEGACY)))
            torch.cuda.synchronize()
            want = torch.full_like(U, 9.0)
            want[lo * Np:hi * Np] = a[lo * Np:hi * Np]
            assert torch.equal(c, want), (lo, hi)


def test_nonlinear_forms_keep_the_quadrature_kernels():
    for nu2 in (0.0, 0.5):
        op, g, dom, cod = make((3, 3, 3), 2, [O.SIPLaplace(4.0, "u", nu0=1.0, nu2=nu2)], (True, True, True),
                               quad=O.QuadOrderFunc.NonLinear(3))
        with op.GetEvaluatorEx(dom, None, cod) as ev:
            assert (ev.kernel_info(0)[0] == 5) == (nu2 == 0.0)


@pytest.mark.parametrize("n", [(2, 1, 3), (3, 2)], ids=["3d", "2d"])
@pytest.mark.parametrize("kind", ["diffusion", "transport"])
def test_modal_volume_terms_of_small_variations_on_a_large_mean(n, kind):
    """Equal cells with even modes only: the jumps vanish exactly and the derivatives do not see the
    mean, so products of a field 2^40 + O(1) are accurate relative to the O(1) part."""
    import torch
    dim = len(n)
    for k in (2, 3, 4):
        comp = O.SIPLaplace(4.0, "u", nu0=0.3) if kind == "diffusion" else O.ScalarTransportFlux([0.7, -0.4, 0.3][:dim], "u")
        op, g, dom, cod = make(n, k, [comp], (True,) * dim)
        desc = (op.descriptor([k], [k], dim), g.desc())
        # modes by total degree, then the first exponents
        exps = [e for d in range(k + 1) for e in np.ndindex(*(k + 1,) * dim) if sum(e) == d]
        r = np.random.default_rng(k)
        c = np.array([0.0 if any(i & 1 for i in e) else r.uniform(0.5, 1.0) for e in exps])
        c[0] += 2.0 ** 40
        U = np.tile(c, g.NoOfCells)
        u = torch.from_numpy(U).cuda()
        with op.GetEvaluatorEx(dom, None, cod) as ev:
            assert ev.kernel_info(0)[0] == 5
            if kind == "transport":
                pairs = [(ev.vjp(u, u), orc.vjp(*desc, U, U))]
            else:     # a symmetric operator: J^T w = J w
                out = torch.zeros_like(u)
                ev.Evaluate(1.0, 0.0, out, u)
                jvp = orc.jvp(*desc, U, U)
                pairs = [(out, orc.evaluate(*desc, U)), (ev.jvp(u, u), jvp), (ev.vjp(u, u), jvp)]
            for got, want in pairs:
                assert np.linalg.norm(want) < 1e4     # the mean does not enter
                assert rel(got.cpu().numpy(), want) <= TOL, k
