"""Nonlinear diffusion (SIP with nu(u)) on the face-once block kernel: residual, JVP and VJP against
the oracle for every degree and rule with an instance, at the sizes where blocks are cut (one
cell, two periodic cells, sizes around the block extents), in both cell orders, with every
boundary kind, on cell ranges and on vectors that start at an odd double."""
import ctypes

import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the parity bar of every FP64 kernel against the oracle

RULES = [(1, 2), (1, 3), (2, 3), (2, 4), (2, 5), (3, 4), (3, 5), (3, 7), (4, 5), (4, 7), (4, 9)]
CASES = [((1, 1, 2), (True, True, True), 0), ((5, 3, 9), (False, False, False), 0), ((4, 7, 5), (True, False, True), 1),
         ((9, 2, 6), (False, True, False), 2)]


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def make(n, k, q, periodic, kind, order=C.CELLS_GENERATOR):
    nodes = [np.linspace(0.1 * d, 0.1 * d + 1.0 + 0.3 * d, v + 1) for d, v in enumerate(n)]
    g = O.Cartesian3DGrid(*nodes, *periodic, cell_order=order)
    op = O.DifferentialOperator(["u"], [], ["R"], O.QuadOrderFunc.FixedOrder(2 * q - 1))
    if kind == 0:
        comps = [O.SIPLaplace(4.0, "u", nu0=1.0, nu2=0.7)]
    elif kind == 1:
        comps = [O.ScalarTransportFlux([0.7, -0.4, 0.3], "u"), O.ConstantSource(1.3, "u"),
                 O.SIPLaplace(4.0, "u", nu0=0.3, nu2=-0.4, g0=0.2, g1=(0.5, -0.3, 0.1), g2=(0.4, 0.2, -0.6))]
    else:
        comps = [O.ScalarTransportFlux([-0.7, 0.4, -0.3], "u"), O.SIPLaplace(4.0, "u", nu0=0.5, nu2=0.3, dirichlet=False)]
    for c in comps:
        op.EquationComponents["R"].Add(c)
    op.Commit()
    return op, g, [O.DGField(g, k, "u")], [O.DGField(g, k, "R")]


@pytest.mark.parametrize("k,q", RULES)
@pytest.mark.parametrize("n,periodic,kind", CASES, ids=["1x1x2", "5x3x9", "4x7x5", "9x2x6"])
def test_sip_blocks_match_oracle(n, periodic, kind, k, q):
    import torch
    for order in (C.CELLS_GENERATOR, C.CELLS_GLOBALID):
        op, g, dom, cod = make(n, k, q, periodic, kind, order)
        desc = (op.descriptor([k], [k], 3), g.desc())
        r = np.random.default_rng(k)
        U, V, prev = (r.uniform(-1, 1, g.NoOfCells * dom[0].Np) for _ in range(3))
        pad = torch.zeros(2 * U.size + 1, dtype=torch.float64, device="cuda")
        u, out = pad[1:U.size + 1], pad[U.size + 1:]     # u starts at an odd double
        u.copy_(torch.from_numpy(U))
        v = torch.from_numpy(V).cuda()
        out.copy_(torch.from_numpy(prev))
        with op.GetEvaluatorEx(dom, None, cod) as ev:
            assert [ev.kernel_info(m)[0] for m in range(3)] == [6, 6, 6]
            ev.Evaluate(0.7, 0.3, out, u)
            ref = orc.evaluate(*desc, U)
            torch.cuda.synchronize()
            assert rel((out.cpu().numpy() - 0.3 * prev) / 0.7, ref) <= TOL
            assert rel(ev.jvp(u, v).cpu().numpy(), orc.jvp(*desc, U, V)) <= TOL
            assert rel(ev.vjp(u, v).cpu().numpy(), orc.vjp(*desc, U, V)) <= TOL


def test_sip_blocks_cell_ranges():
    import torch
    op, g, dom, cod = make((6, 5, 7), 2, 5, (False, True, False), 1)
    N, Np = g.NoOfCells * dom[0].Np, dom[0].Np
    r = np.random.default_rng(3)
    U, V = (torch.from_numpy(r.uniform(-1, 1, N)).cuda() for _ in range(2))
    with op.GetEvaluatorEx(dom, None, cod) as ev:
        for mode in range(3):
            whole = torch.zeros_like(U)
            args = (C.ptr(U), C.ptr(V) if mode else None)
            st = ctypes.c_void_p(C.CUDA_STREAM_LEGACY)
            C.check(C.lib().bosss_b200_apply_device(ev.handle, mode, 1.0, 0.0, *args, C.ptr(whole), 0.0, 0, g.NoOfCells, st))
            for lo, hi in ((0, 1), (34, 36), (13, 171)):
                c = torch.full_like(U, 9.0)
                C.check(C.lib().bosss_b200_apply_device(ev.handle, mode, 1.0, 0.0, *args, C.ptr(c), 0.0, lo, hi, st))
                torch.cuda.synchronize()
                want = torch.full_like(U, 9.0)
                want[lo * Np:hi * Np] = whole[lo * Np:hi * Np]
                assert torch.equal(c, want), (mode, lo, hi)


@pytest.mark.parametrize("k,q,small,large", [(3, 7, (8, 37, 1), (11, 27, 1)), (4, 7, (16, 37, 1), (1, 593, 1)),
                                             (4, 9, (8, 37, 1), (11, 27, 1))])
def test_products_on_both_sides_of_the_small_grid_rule(k, q, small, large):
    """J v and J^T w with 7 or 9 nodes run on the generic tiles as long as these fit one wave (296 or 592
    cells): its bits below the line, blocks that match the oracle from there on."""
    import torch
    for n in (small, large):
        op, g, dom, cod = make(n, k, q, (True, False, True), 1)
        desc = (op.descriptor([k], [k], 3), g.desc())
        r = np.random.default_rng(k)
        U, V = (r.uniform(-1, 1, g.NoOfCells * dom[0].Np) for _ in range(2))
        u, v = torch.from_numpy(U).cuda(), torch.from_numpy(V).cuda()
        got = []
        for kernel in (C.KERNEL_AUTO, C.KERNEL_GENERIC):
            with op.GetEvaluatorEx(dom, None, cod, kernel=kernel) as ev:
                got.append([ev.jvp(u, v), ev.vjp(u, v)])
        assert all(torch.equal(a, b) for a, b in zip(*got)) == (n == small)
        for t, f in zip(got[0], (orc.jvp, orc.vjp)):
            assert rel(t.cpu().numpy(), f(*desc, U, V)) <= TOL
