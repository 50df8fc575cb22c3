"""3D Euler / HLLC on the face-once block kernel: residual, JVP and VJP against the oracle for every
degree, at the sizes where blocks are cut (one cell, two periodic cells, sizes around the block
extents), in both cell orders, with shock-like jumps (every HLLC branch), on cell ranges and on
vectors that start at an odd double."""
import ctypes

import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from bosss_b200 import problems as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the parity bar of every FP64 kernel against the oracle

SIZES = [(1, 1, 1), (2, 1, 3), (5, 4, 9), (3, 7, 2)]


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def make(n, k, order, seed, speed):
    nodes = [np.linspace(0.0, 1.0 + 0.2 * d, v + 1) for d, v in enumerate(n)]
    g = O.Cartesian3DGrid(*nodes, True, True, True, cell_order=order)
    ref = P.euler3d(n=2, k=k).op
    dom = [O.DGField(g, k, s) for s in ref.DomainVar]
    cod = [O.DGField(g, k, s) for s in ref.CodomainVar]
    r = np.random.default_rng(seed)
    J, Q = g.NoOfCells, (k + 1) ** 3
    # cell-wise velocity offsets of `speed` reach the supersonic branches of both signs
    rho = 1.0 + 0.1 * r.uniform(-1, 1, (J, Q))
    vel = 0.2 * r.uniform(-1, 1, (3, J, Q)) + speed * r.uniform(-1, 1, (3, J, 1))
    p = 1.0 + 0.1 * r.uniform(-1, 1, (J, Q)) + 0.5 * r.uniform(0, 1, (J, 1))
    E = p / 0.4 + 0.5 * rho * (vel ** 2).sum(0)
    h = [(b - a) / v for a, b, v in zip(g.lo, g.hi, g.n)]
    U = np.stack([P.project_nodal(3, k, k + 1, h, f) for f in (rho, rho * vel[0], rho * vel[1], rho * vel[2], E)], 1)
    return ref, g, dom, cod, U.ravel()


@pytest.mark.parametrize("speed", [0.1, 3.0], ids=["subsonic", "supersonic"])
@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", SIZES, ids=lambda n: "x".join(map(str, n)))
def test_euler_blocks_match_oracle(n, k, speed):
    import torch
    for order in (C.CELLS_GENERATOR, C.CELLS_GLOBALID):
        op, g, dom, cod, U = make(n, k, order, 7 * k + len(n), speed)
        desc = (op.descriptor([k] * 5, [k] * 5, 3), g.desc())
        r = np.random.default_rng(k)
        V, prev = (r.uniform(-1, 1, U.size) for _ in range(2))
        pad = torch.zeros(2 * U.size + 1, dtype=torch.float64, device="cuda")
        u, out = pad[1:U.size + 1], pad[U.size + 1:]     # u starts at an odd double
        u.copy_(torch.from_numpy(U))
        v = torch.from_numpy(V).cuda()
        out.copy_(torch.from_numpy(prev))
        with op.GetEvaluatorEx(dom, None, cod) as ev:
            assert [ev.kernel_info(m)[0] for m in range(3)] == [7, 7, 7]
            ev.Evaluate(0.7, 0.3, out, u)
            ref = 0.3 * prev + 0.7 * orc.evaluate(*desc, U)
            torch.cuda.synchronize()
            assert rel(out.cpu().numpy(), ref) <= TOL
            assert rel(ev.jvp(u, v).cpu().numpy(), orc.jvp(*desc, U, V)) <= TOL
            assert rel(ev.vjp(u, v).cpu().numpy(), orc.vjp(*desc, U, V)) <= TOL


def test_euler_blocks_cell_ranges():
    import torch
    op, g, dom, cod, U = make((6, 5, 7), 2, C.CELLS_GENERATOR, 5, 0.5)
    npc = 5 * dom[0].Np
    u, v = torch.from_numpy(U).cuda(), torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, U.size)).cuda()
    st = ctypes.c_void_p(C.CUDA_STREAM_LEGACY)
    with op.GetEvaluatorEx(dom, None, cod) as ev:
        for mode in range(3):
            whole = torch.zeros_like(u)
            args = (C.ptr(u), C.ptr(v) if mode else None)
            C.check(C.lib().bosss_b200_apply_device(ev.handle, mode, 1.0, 0.0, *args, C.ptr(whole), 0.0, 0, g.NoOfCells, st))
            for lo, hi in ((0, 1), (34, 36), (13, 171)):
                c = torch.full_like(u, 9.0)
                C.check(C.lib().bosss_b200_apply_device(ev.handle, mode, 1.0, 0.0, *args, C.ptr(c), 0.0, lo, hi, st))
                torch.cuda.synchronize()
                want = torch.full_like(u, 9.0)
                want[lo * npc:hi * npc] = whole[lo * npc:hi * npc]
                assert torch.equal(c, want), (mode, lo, hi)


@pytest.mark.parametrize("speed", [0.1, 3.0], ids=["subsonic", "supersonic"])
@pytest.mark.parametrize("k", [1, 3])
def test_densities_whose_product_leaves_the_double_range(k, speed):
    """rho -> A rho, u -> B u, p -> A B^2 p is an exact symmetry; with powers of two every operation of
    the kernels scales exactly, so all three products give the scaled bits."""
    import torch
    op, g, dom, cod, U = make((3, 4, 5), k, C.CELLS_GENERATOR, 11 + k, speed)
    J, A, B = g.NoOfCells, 2.0 ** 515, 2.0 ** -10      # rho_A rho_B about 2^1030, momentum^2 below 2^1016
    su = np.array([A, A * B, A * B, A * B, A * B * B])[None, :, None]
    sf = su * B
    U = U.reshape(J, 5, -1)
    r = np.random.default_rng(k)
    V, W = r.uniform(-1, 1, U.shape), r.uniform(-1, 1, U.shape)
    res = []
    with op.GetEvaluatorEx(dom, None, cod) as ev:
        for s, f in ((1.0, 1.0), (su, sf)):
            u, v, w = (torch.from_numpy(np.ascontiguousarray(t).ravel()).cuda() for t in (U * s, V * s, W / f))
            out = torch.zeros_like(u)
            ev.Evaluate(1.0, 0.0, out, u)
            res.append([t.cpu().numpy().reshape(U.shape) for t in (out, ev.jvp(u, v), ev.vjp(u, w))])
    for a, b, s in zip(res[0], res[1], (sf, sf, 1.0 / su)):
        assert np.isfinite(a).all() and np.array_equal(a * s, b)


@pytest.mark.parametrize("value", [np.nan, 0.0], ids=["nan", "vacuum"])
@pytest.mark.parametrize("speed", [0.1, 3.0], ids=["subsonic", "supersonic"])
def test_a_bad_density_reaches_the_cells_it_reaches_on_the_slab_kernel(speed, value):
    """The flux reads the upwind state only where the waves run one way: a NaN or vanishing density of a
    cell reaches the same cells as on the quadrature slab kernel."""
    import torch
    k = 2
    op, g, dom, cod, U = make((5, 4, 6), k, C.CELLS_GENERATOR, 3, speed)
    J = g.NoOfCells
    V = np.random.default_rng(5).uniform(-1, 1, U.size)
    U = U.reshape(J, 5, -1)
    U[J // 2, 0, :] = 0.0
    U[J // 2, 0, 0] = value
    u, v = torch.from_numpy(U.ravel()).cuda(), torch.from_numpy(V).cuda()
    sets = []
    for kernel in (C.KERNEL_AUTO, C.KERNEL_SLAB):
        with op.GetEvaluatorEx(dom, None, cod, kernel=kernel) as ev:
            out = torch.zeros_like(u)
            ev.Evaluate(1.0, 0.0, out, u)
            sets.append([np.nonzero(~np.isfinite(t.cpu().numpy().reshape(J, -1)).all(axis=1))[0].tolist()
                         for t in (out, ev.jvp(u, v), ev.vjp(u, v))])
    assert sets[0] == sets[1]


@pytest.mark.parametrize("k", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(10, 5, 4), (18, 17, 1), (9, 4, 3)], ids=lambda n: "x".join(map(str, n)))
def test_euler_bits_do_not_depend_on_the_place_in_a_block(n, k):
    """Ranges of planes cut the blocks differently; every cell keeps the bits of the whole-grid call, as
    partitioned grids and the chunks of the host path rely on."""
    import torch
    op, g, dom, cod, U = make(n, k, C.CELLS_GENERATOR, 23, 0.1)
    plane, npc = n[1] * n[2], 5 * dom[0].Np
    u, v = torch.from_numpy(U).cuda(), torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, U.size)).cuda()
    st = ctypes.c_void_p(C.CUDA_STREAM_LEGACY)
    with op.GetEvaluatorEx(dom, None, cod) as ev:
        for mode in range(3):
            args = (C.ptr(u), C.ptr(v) if mode else None)

            def cells(lo, hi):
                out = torch.zeros_like(u)
                C.check(C.lib().bosss_b200_apply_device(ev.handle, mode, 1.0, 0.0, *args, C.ptr(out), 0.0, lo, hi, st))
                torch.cuda.synchronize()
                return out[lo * npc:hi * npc]

            whole = cells(0, g.NoOfCells)
            for size in (1, 2, 3, 5):
                for p in range(0, n[0], size):
                    lo, hi = p * plane, min(p + size, n[0]) * plane
                    assert torch.equal(cells(lo, hi), whole[lo * npc:hi * npc]), (mode, size, p)


@pytest.mark.parametrize("n,slab", [((12, 37, 4), True), ((1777, 1, 1), False)], ids=["1776_cells", "1777_cells"])
def test_small_grid_rule_of_the_quadratic_adjoint(n, slab):
    """J^T w for k = 2 runs on the slab tiles as long as these fit one wave (1776 cells): its bits below
    the line, blocks that match the oracle from there on."""
    import torch
    op, g, dom, cod, U = make(n, 2, C.CELLS_GENERATOR, 9, 0.5)
    W = np.random.default_rng(2).uniform(-1, 1, U.size)
    u, w = torch.from_numpy(U).cuda(), torch.from_numpy(W).cuda()
    got = []
    for kernel in (C.KERNEL_AUTO, C.KERNEL_SLAB):
        with op.GetEvaluatorEx(dom, None, cod, kernel=kernel) as ev:
            got.append(ev.vjp(u, w))
    assert torch.equal(*got) == slab
    assert rel(got[0].cpu().numpy(), orc.vjp(op.descriptor([2] * 5, [2] * 5, 3), g.desc(), U, W)) <= TOL
