"""Cut items and the interface term at every degree: the species residuals with linear and with
solution-dependent viscosity, transport, a sphere that cuts the domain boundary (cut boundary
faces with Dirichlet data) and both cut-rule families, against the oracle with the same rules."""
import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TOL = 1e-12   # the parity bar of every FP64 kernel against the oracle


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def ops(nu2):
    out = []
    for mu in (1.0, 10.0):
        op = O.DifferentialOperator(["u"], [], ["R"], O.QuadOrderFunc.FixedOrder(0))
        op.EquationComponents["R"].Add(O.SIPLaplace(4.0, "u", nu0=mu, nu2=nu2 * mu, g0=0.2, g1=(0.5, -0.3, 0.1),
                                                    g2=(0.4, 0.2, -0.6)))
        op.EquationComponents["R"].Add(O.ConstantSource(1.0, "u"))
        op.EquationComponents["R"].Add(O.ScalarTransportFlux([0.7, -0.4, 0.3], "u"))
        out.append(op)
    return out


@pytest.mark.parametrize("rule", [C.XDG_RULE_MOMENT_FITTING, C.XDG_RULE_SAYE], ids=["fitted", "saye"])
@pytest.mark.parametrize("nu2", [0.0, 0.3], ids=["linear", "nonlinear"])
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_cut_items_match_oracle(k, nu2, rule):
    n = 6
    nodes = np.linspace(-1.0, 1.0, n + 1)
    g = O.Cartesian3DGrid(nodes, nodes, nodes, False, False, False)
    opA, opB = ops(nu2)
    for op in (opA, opB):
        op.QuadOrderFunction = O.QuadOrderFunc.FixedOrder(2 * k + 1)
        op.Commit()
    center = (0.55, 0.03, -0.04)   # the sphere reaches the face x = 1
    N = g.NoOfCells * O.np_of(3, k)
    r = np.random.default_rng(10 * k)
    U = [0.1 * r.uniform(-1, 1, N) for _ in range(2)]
    with O.XdgEvaluator(opA, opB, g, k, center, 0.6, rule=rule) as X:
        for s, op in enumerate((opA, opB)):
            R = X.rules(s)
            assert (R["info"][:, 1] == 2).any() and (R["info"][:, 1] == 3).any()
            ref = orc.xdg_evaluate(op.descriptor([k], [k], 3), g.desc(), R, U[s], length_scales=X.length_scales(s))
            out = np.full(N, 3.0)
            X.Evaluate(s, 1.0, 0.0, out, U[s])
            assert rel(out, ref) <= TOL, (s, rel(out, ref))
