"""One batch against the oracle where the step's kernels change form: score rows at the widths of the loss kernels' register
rows (128, 256, 512, 1024), the fused score kernel's narrow form (up to 128 score columns a side), column tiles that do not divide the
gradient's width, chunks and column counts of one, and operator rows above 1024 floats."""
import numpy as np
import pytest

from oracle import pbg_step as O
from test_gpu_step import RTOL, _close, _random_case, _tier_tolerance

pytestmark = pytest.mark.gpu


def _run(case, precision):
    from b200_util import Rig
    c, ocfg, ost, batches = case
    rig = Rig.from_oracle_state(c, ost, precision=precision)
    W0 = ost.W_lhs.copy()
    b = batches[0]
    want = O.train_batch(ocfg, ost, *b)
    got = rig.trainer.process_one_batch(rig.model, rig.edges(b[0], b[1], b[2]), b[3], b[4])
    assert got.metrics["loss"] == pytest.approx(want["loss"], rel=RTOL if precision != "bf16x3" else 10 * RTOL)
    step = float(np.abs(ost.W_lhs - W0).max())
    _close(rig.W_lhs.cpu().numpy(), ost.W_lhs, atol=max(1e-6, RTOL * step), what="W")
    _close(rig.G("lhs"), ost.G_lhs, atol=1e-8, what="G")
    if ost.theta_rhs is not None:
        _close(rig.theta("rhs"), ost.theta_rhs, atol=1e-6, what="theta_rhs")


@pytest.mark.parametrize("cols", [128, 129, 256, 257, 512, 513, 1024, 1025])
@pytest.mark.parametrize("comp,loss", [("dot", "ranking"), ("dot", "logistic"), ("l2", "softmax")])
def test_score_rows_at_the_loss_kernels_widths(cols, comp, loss):
    nb = cols // 2
    _run(_random_case(5, 24, 4000, 2 * nb + 3, nb, cols - nb, "none", comp, loss), "tf32x3")


@pytest.mark.parametrize("tier", ["bf16x6", "bf16x3"])
@pytest.mark.parametrize("nb,nu", [(1, 1), (64, 64), (64, 65), (100, 28), (100, 29), (128, 1)])
def test_fused_scores_at_the_narrow_form_s_edge(nb, nu, tier, monkeypatch):
    monkeypatch.setenv("PBG_FUSED", "1")
    with _tier_tolerance(tier):
        _run(_random_case(6, 100, 4000, 5 * nb + 1, nb, nu, "none", "dot", "softmax"), tier)


@pytest.mark.parametrize("precision", ["fp32", "tf32x3", "bf16x6", "bf16x3"])
@pytest.mark.parametrize("D,nb,nu", [(400, 260, 37), (260, 129, 0), (516, 1, 300), (776, 100, 1)])
def test_column_tiles_of_both_gradients(D, nb, nu, precision):
    with _tier_tolerance(precision):
        _run(_random_case(7, D, 3000, 2 * nb + 1, nb, nu, "diagonal", "dot", "softmax", dyn=True, R=9), precision)


@pytest.mark.parametrize("D", [1024, 1028])
def test_operator_rows_of_wide_models(D):
    _run(_random_case(8, D, 2000, 300, 50, 20, "translation", "dot", "softmax", dyn=True, R=4, zipf=True), "tf32x3")


@pytest.mark.parametrize("D", [4, 64, 68, 128, 132, 192, 196, 256, 260])
@pytest.mark.parametrize("N,nb,nu", [(9, 30, 5), (150, 40, 11), (6000, 50, 50)])
def test_update_rows_at_the_half_warp_kernels_widths(D, N, nb, nu):
    """Hub rows only, short rows across tiles and hubs, and rows of a single slot, at the edges of a half-warp's row."""
    _run(_random_case(9, D, N, 5 * nb + 2, nb, nu, "none", "dot", "softmax", zipf=N > 10), "tf32x3")


@pytest.mark.parametrize("precision", ["tf32x3", "bf16x6"])
@pytest.mark.parametrize("D,R,k", [(36, 5, 1), (100, 900, 4), (260, 40, 3)])
def test_sibling_launches_wave_after_wave(D, R, k, precision):
    """Dynamic relations: the two gradients, and the tile and hub kernels of embedding and operator rows, run into one another.
    Several waves in one call (k >= 2: halves on two streams), against the oracle, and the same bits every time."""
    import torch
    from b200_util import Rig
    c, ocfg, ost, batches = _random_case(10, D, 700, 310, 30, 20, "diagonal", "dot", "softmax", dyn=True, R=R, zipf=True, nbatches=2 * k + 1)
    start = [ost.W_lhs.copy(), ost.G_lhs.copy(), ost.theta_rhs.copy(), ost.theta_lhs.copy()]
    lhs, rhs, rel = (np.concatenate([b[i] for b in batches]) for i in range(3))
    runs = []
    for _ in range(3):
        rig = Rig.from_oracle_state(c, ost, precision=precision, k=k)
        nat = rig.trainer._context(rig.model, 310)
        ul, ur = (torch.stack([nat._uniform(b[i], "cuda") for b in batches]).contiguous() for i in (3, 4))
        t = lambda a: torch.tensor(a).cuda()
        rig.trainer.train_batches(rig.model, t(lhs), t(rhs), t(rel), [(i * 310, 310, 0) for i in range(len(batches))], ul, ur)
        runs.append((rig.W_lhs.cpu().numpy(), rig.G("lhs"), rig.theta("rhs"), rig.theta("lhs"), rig.acc("rhs"), rig.acc("lhs")))
    for other in runs[1:]:
        for a, b in zip(runs[0], other):
            np.testing.assert_array_equal(a, b)
    nwaves = -(-len(batches) // k)
    sizes = [len(batches) // nwaves + (w < len(batches) % nwaves) for w in range(nwaves)]      # dealt evenly
    for n in sizes:
        O.train_wave(ocfg, ost, batches[:n])
        batches = batches[n:]
    with _tier_tolerance(precision):
        for got, want, was, what in zip(runs[0], (ost.W_lhs, ost.G_lhs, ost.theta_rhs, ost.theta_lhs), start, ("W", "G", "theta_rhs", "theta_lhs")):
            _close(got, want, atol=max(1e-6, RTOL * float(np.abs(want - was).max())), what=what)
