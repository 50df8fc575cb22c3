"""Non-finite coefficients on the modal kernel reach the cells that they reach through the quadrature
kernels, and no others: the upwind flux takes one side's value, so a NaN or Inf does not travel
upwind, and a source alone reads no coefficients (residual, J v; the adjoint's jump has both sides)."""
import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O

pytestmark = pytest.mark.gpu


def make(n, k, comps, periodic):
    nodes = [np.linspace(0.0, 1.0 + 0.3 * d, v + 1) for d, v in enumerate(n)]
    g = (O.Cartesian2DGrid if len(n) == 2 else O.Cartesian3DGrid)(*nodes, *periodic)
    op = O.DifferentialOperator(["u"], [], ["R"], O.QuadOrderFunc.Linear())
    for c in comps:
        op.EquationComponents["R"].Add(c)
    op.Commit()
    return op, g, [O.DGField(g, k, "u")], [O.DGField(g, k, "R")]


def bad_cells(t, cells):
    return np.nonzero(~np.isfinite(t.cpu().numpy().reshape(cells, -1)).all(axis=1))[0].tolist()


VEL = (0.7, -0.4, 0.0)
COMPS = {"transport": lambda d: [O.ScalarTransportFlux(VEL[:d], "u")],
         "against": lambda d: [O.ScalarTransportFlux([-v for v in VEL[:d]], "u")],
         "transport_source": lambda d: [O.ScalarTransportFlux(VEL[:d], "u"), O.ConstantSource(1.3, "u")],
         "advdiff": lambda d: [O.ScalarTransportFlux(VEL[:d], "u"), O.SIPLaplace(4.0, "u", nu0=0.3)],
         "source": lambda d: [O.ConstantSource(1.3, "u")]}


@pytest.mark.parametrize("value", [np.nan, np.inf], ids=["nan", "inf"])
@pytest.mark.parametrize("kind", sorted(COMPS))
@pytest.mark.parametrize("n,periodic", [((4, 5, 3), (True, True, True)), ((5, 4, 3), (False, True, False)),
                                        ((5, 6), (True, True))], ids=["periodic", "bounded", "2d"])
def test_nonfinite_values_reach_the_same_cells(n, periodic, kind, value):
    import torch
    cells = int(np.prod(n))
    for k in (1, 2, 4):
        op, g, dom, cod = make(n, k, COMPS[kind](len(n)), periodic)
        Np = dom[0].Np
        r = np.random.default_rng(k)
        U = r.uniform(-1, 1, cells * Np)
        bad = U.copy()
        bad[(cells // 2) * Np + int(r.integers(Np))] = value
        u, v = torch.from_numpy(U).cuda(), torch.from_numpy(bad).cuda()
        sets = []
        for kernel in (C.KERNEL_AUTO, C.KERNEL_GENERIC):
            with op.GetEvaluatorEx(dom, None, cod, kernel=kernel) as ev:
                assert (ev.kernel_info(0)[0] == 5) == (kernel == C.KERNEL_AUTO)
                out = torch.zeros_like(u)
                ev.Evaluate(1.0, 0.0, out, v)
                sets.append([bad_cells(t, cells) for t in (out, ev.jvp(u, v), ev.vjp(u, v))])
        assert sets[0] == sets[1], (k, sets)


@pytest.mark.parametrize("kernel", [C.KERNEL_AUTO, C.KERNEL_GENERIC], ids=["modal", "generic"])
def test_nan_check_refuses_products_at_a_nonfinite_state(kernel):
    """With the NaN check on, J v and J^T w of a diffusion operator at a state with a NaN or Inf are
    refused, on the modal kernel too, which does not read the state for them."""
    n, k = (3, 4, 2), 2
    op, g, dom, cod = make(n, k, COMPS["advdiff"](3), (True, False, True))
    U = np.random.default_rng(1).uniform(-1, 1, g.NoOfCells * dom[0].Np)
    with op.GetEvaluatorEx(dom, None, cod, kernel=kernel, check_nan=True) as ev:
        ev.jvp(U, U)
        ev.vjp(U, U)
        for value in (np.nan, np.inf):
            bad = U.copy()
            bad[77] = value
            for product in (ev.jvp, ev.vjp):
                with pytest.raises(C.BosssError) as e:
                    product(bad, U)
                assert e.value.code == C.ERR_NAN
