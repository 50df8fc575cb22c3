"""The work queue and the class launches of the batch (nonlinear instances and explicit kernel
selectors; linear batches run on the modal kernel): every schedule against the oracle and the single
instances, the captured step, and the autotuner's table."""
import numpy as np
import pytest

from bosss_b200 import _capi as C
from bosss_b200 import operator as O
from bosss_b200 import problems as P
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def linear_batch():
    return P.batched_advection_diffusion(n_instances=6, seed=77, sizes=(3, 4, 5), degrees=(1, 2, 3))


def nonlinear_batch():
    """The same shape of batch; every second instance has nu(u) = nu0 + nu2 u^2."""
    probs = linear_batch()
    for i, p in enumerate(probs):
        if i % 2 == 0:
            op = O.DifferentialOperator(["u"], [], ["R"], O.QuadOrderFunc.Linear())
            op.EquationComponents["R"].Add(O.ScalarTransportFlux(p.config["velocity"], "u"))
            op.EquationComponents["R"].Add(O.SIPLaplace(4.0, "u", nu0=0.3, nu2=0.2))
            op.Commit()
            p.op = op
    return probs


def vectors(probs):
    import torch
    U = torch.from_numpy(np.concatenate([p.U for p in probs])).cuda()
    W = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, U.numel())).cuda()
    return U, W, torch.zeros_like(U), torch.zeros_like(U)


@pytest.mark.parametrize("later", ["nonlinear", "generic", "slab"])
def test_tuning_a_linear_batch_records_nothing_for_queue_batches(tmp_path, later):
    """The modal path has nothing to time: the table keeps what it held, and a queue batch of the same
    classes is tuned when it comes."""
    table = tmp_path / "tiles.txt"
    table.write_text("phys9_D3_K9_Q9 4\n")
    probs = linear_batch()
    with O.BatchEvaluator(probs) as b:
        b.autotune(*vectors(probs), str(table))
    assert table.read_text().split() == ["phys9_D3_K9_Q9", "4"]
    probs = nonlinear_batch() if later == "nonlinear" else probs
    kernel = {"nonlinear": C.KERNEL_AUTO, "generic": C.KERNEL_GENERIC, "slab": C.KERNEL_SLAB}[later]
    with O.BatchEvaluator(probs, kernel=kernel) as b:
        b.autotune(*vectors(probs), str(table))
    text = table.read_text()
    for k in {p.dom[0].degree for p in probs}:
        assert "_D3_K%d_Q%d" % (k, k + 1) in text      # tuned and recorded
    assert text.splitlines()[-1].split()[0] == "schedule"


def test_linear_batches_build_no_queue():
    """Work items and class lists (24 bytes per tile, mode and list) are not built for a batch that
    never reads them."""
    import torch
    probs = [P.advection_diffusion3d(n=32, k=4, seed=5, velocity=(0.3, -0.2, 0.5))] * 32    # 1.05e6 cells

    def device_bytes():
        free0 = torch.cuda.mem_get_info()[0]
        with O.BatchEvaluator(probs):
            return free0 - torch.cuda.mem_get_info()[0]

    device_bytes()                    # kernels loaded
    assert device_bytes() <= 6 << 20  # the lists take 10 MB here


KINDS = {"generic": (linear_batch, C.KERNEL_GENERIC), "slab": (linear_batch, C.KERNEL_SLAB),
         "nonlinear": (nonlinear_batch, C.KERNEL_AUTO)}


@pytest.mark.parametrize("schedule", ["classes", "lpt", "fifo"])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_queue_schedules_match_oracle_and_single_instances(tmp_path, kind, schedule):
    import torch
    make, kernel = KINDS[kind]
    probs = make()
    U, W, R, G = vectors(probs)
    table = tmp_path / "tiles.txt"
    table.write_text("schedule %s\n" % schedule)
    with O.BatchEvaluator(probs, kernel=kernel) as b:
        b.autotune(U, W, R, G, str(table))
        assert b.tiles(1, 2)[1] == schedule
        out = [b.evaluate(m, U, None if m == C.MODE_RESIDUAL else W) for m in range(3)]
        torch.cuda.synchronize()
        off = b.dom_offsets
    for i, p in enumerate(probs):
        sl = slice(int(off[i]), int(off[i + 1]))
        got = [t[sl].cpu().numpy() for t in out]
        w = W[sl].cpu().numpy()
        ref = [orc.evaluate(*p.descs(), p.U), orc.jvp(*p.descs(), p.U, w), orc.vjp(*p.descs(), p.U, w)]
        for a, r in zip(got, ref):
            assert rel(a, r) <= 1e-12
        if kind != "nonlinear":       # the tiles of the single-grid kernel
            with p.evaluator(kernel=kernel) as ev:
                single = np.zeros(p.n_dofs)
                ev.Evaluate(1.0, 0.0, single, p.U)
                for a, r in zip(got, (single, ev.jvp(p.U, w), ev.vjp(p.U, w))):
                    assert rel(a, r) <= 1e-13


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_queue_graph_replay_and_autotune(tmp_path, kind):
    import torch
    make, kernel = KINDS[kind]
    probs = make()
    U, W, R, G = vectors(probs)
    table = str(tmp_path / "tiles.txt")
    with O.BatchEvaluator(probs, kernel=kernel) as b:
        Rd, Gd = b.evaluate(C.MODE_RESIDUAL, U), b.evaluate(C.MODE_VJP, U, W)
        b.autotune(U, W, R, G, table)
        b.capture(U, W, R, G)
        R.zero_()
        G.zero_()
        b.replay()
        torch.cuda.synchronize()
        assert torch.equal(R, Rd) and torch.equal(G, Gd)
        tiles = {k: b.tiles(k, k + 1) for k in (1, 2, 3)}
    with O.BatchEvaluator(probs, kernel=kernel) as b2:      # reads the table instead of timing again
        b2.autotune(U, W, R, G, table)
        assert {k: b2.tiles(k, k + 1) for k in tiles} == tiles
