"""The one-kernel path of small waves (pbg_chunk.cu) against the oracle, at the edges of its tiles (16 score rows, 32 gradient
rows, 128 columns and k-values, 128 floats per lane group), and the separate kernels where the default has become that path."""
import numpy as np
import pytest
import torch

from golden_util import load_step, step_fixture_names
from oracle import pbg_step as O
import test_gpu_step as steps
import test_gpu_step_edges as edges

pytestmark = pytest.mark.gpu

SHAPES = [
    # D, B, nb, nu, op, comp, loss, dyn
    (4, 33, 16, 1, "none", "dot", "softmax", False),                   # one score tile, a last chunk of one edge
    (128, 130, 17, 15, "translation", "cos", "ranking", False),         # a 17th score row, Mm = 32
    (136, 192, 64, 64, "complex_diagonal", "l2", "logistic", False),    # two float4 a lane; the rule's largest tiles
    (256, 150, 65, 63, "diagonal", "squared_l2", "softmax", False),     # a second score tile; k-chunks of 128 and 64
    (100, 200, 50, 50, "none", "cos", "softmax", False),
    (52, 37, 15, 7, "diagonal", "l2", "logistic", False),
    (36, 60, 0, 20, "translation", "dot", "ranking", False),            # uniform negatives only
    (64, 64, 32, 0, "none", "dot", "logistic", False),                  # batch negatives only
    # 250 columns, k-chunks of A beyond 128.  (Not l2 with ranking: a negative that is the edge's own entity has distance 0 in
    # fp64 and up to (4 2^-24 |a|^2)^1/2 = 3e-4 in fp32, its coefficient 1 / 3e-4, and the gradient's two cancelling terms
    # leave 3e3 x 0.1 x 2^-24 = 2e-5 an element, a step of 1e-5 where the other comparators agree to 2e-6.)
    (40, 600, 150, 100, "none", "squared_l2", "ranking", False),
    (24, 70, 20, 10, "complex_diagonal", "dot", "softmax", True),
    (200, 70, 30, 40, "diagonal", "l2", "logistic", True),
    (104, 99, 33, 31, "translation", "cos", "ranking", True),           # a second tile of GQ rows
    (132, 150, 70, 59, "diagonal", "dot", "softmax", False),            # two float4 a lane and a column beyond 128
    (200, 260, 130, 126, "complex_diagonal", "squared_l2", "logistic", False),   # ... and the most columns
    (256, 90, 45, 100, "translation", "cos", "softmax", True),
]


@pytest.mark.parametrize("precision", ["fp32", "tf32x3"])
@pytest.mark.parametrize("D,B,nb,nu,op,comp,loss,dyn", SHAPES)
def test_one_kernel_step_matches_oracle(D, B, nb, nu, op, comp, loss, dyn, precision, monkeypatch):
    """Tolerance: the rtol 1e-4 that both tiers are held to; fp32 sums of fp32 products, whatever the tier."""
    from b200_util import Rig
    monkeypatch.setenv("PBG_CHUNK", "1")
    c, ocfg, ost, batches = steps._random_case(31, D, 400, B, nb, nu, op, comp, loss, dyn, 7 if dyn else 1, zipf=True, w_scale=1.0 if comp == "cos" else 0.1)
    rig = Rig.from_oracle_state(c, ost, precision=precision)
    lhs, rhs, rel, ul, ur = batches[0]
    sc = rig.model(rig.edges(lhs, rhs, rel), ul, ur)
    want = O.score_batch(ocfg, ost, lhs, rhs, rel, ul, ur)
    for k, w in zip(("lhs_pos", "rhs_pos", "lhs_neg", "rhs_neg"), (want[k] for k in ("lhs_pos", "rhs_pos", "lhs_neg", "rhs_neg"))):
        steps._close(getattr(sc, k).cpu().numpy(), w, atol=3e-5 if comp != "l2" else 6e-4, what=k)     # (l2 of equal rows: 0 in fp64)
    ostats = O.train_batch(ocfg, ost, lhs, rhs, rel, ul, ur)
    st = rig.trainer.process_one_batch(rig.model, rig.edges(lhs, rhs, rel), ul, ur)
    assert st.metrics["loss"] == pytest.approx(ostats["loss"], rel=1e-4)
    steps._close(rig.W_lhs.cpu().numpy(), ost.W_lhs, atol=2e-6, what="W")
    steps._close(rig.G("lhs"), ost.G_lhs, atol=1e-7, what="G")
    for side in ("rhs", "lhs"):
        if rig.theta(side) is not None and (dyn or side == "rhs"):
            steps._close(rig.theta(side), ost.theta_rhs if side == "rhs" else ost.theta_lhs, atol=2e-6, what="theta_" + side)


def test_fp32_tier_keeps_its_bits(monkeypatch):
    """The fp32 tier's sums have the order of its separate kernels: the same tables, bit for bit."""
    from b200_util import Rig
    for D, op, comp, loss in ((100, "translation", "cos", "ranking"), (200, "none", "dot", "softmax"), (64, "diagonal", "l2", "logistic")):
        got = []
        for chunk in "01":
            monkeypatch.setenv("PBG_CHUNK", chunk)
            c, ocfg, ost, batches = steps._random_case(8, D, 300, 230, 50, 50, op, comp, loss, zipf=True, w_scale=1.0 if comp == "cos" else 0.1)
            rig = Rig.from_oracle_state(c, ost)
            b = batches[0]
            rig.trainer.process_one_batch(rig.model, rig.edges(b[0], b[1], b[2]), b[3], b[4])
            got.append((rig.W_lhs.cpu().numpy(), rig.G("lhs")))
        for a, b in zip(*got):
            np.testing.assert_array_equal(a, b)


TIERS = steps.PRECISIONS + steps.PLANE_TIERS


@pytest.mark.parametrize("precision", TIERS)
@pytest.mark.parametrize("name", [n for n in step_fixture_names() if load_step(n)[0]["op"] not in ("linear", "affine")])
def test_separate_kernels_on_the_reference_fixtures(name, precision, monkeypatch):
    """The fixtures are small enough for the one-kernel path: the kernels of larger waves on them too."""
    monkeypatch.setenv("PBG_CHUNK", "0")
    with steps._tier_tolerance(precision):
        steps.test_step_matches_reference_fixture(name, precision)
        steps.test_forward_scores_match_reference_fixture(name, precision)


_C1 = steps.BASELINE_SHAPES[0].values
SMALL = ([("waves-of-fixtures", steps.test_wave_of_three_batches_matches_oracle, (n, t), t) for n in ("sequence_3_batches", "sequence_3_batches_dyn_cos") for t in TIERS]
         + [("wave-with-global", steps.test_wave_with_global_embeddings_matches_oracle, (t,), t) for t in TIERS]
         + [("dealt-evenly", steps.test_batches_are_dealt_evenly_to_waves, (), "fp32")]
         + [("C1", steps.test_baseline_shapes_match_oracle, _C1 + (t,), t) for t in TIERS]
         + [("C1", steps.test_single_pass_tf32_is_the_1e3_tier, _C1, "tf32")]
         + [("loss-rows-of-128-%s-%s" % (comp, loss), edges.test_score_rows_at_the_loss_kernels_widths, (128, comp, loss), "tf32x3")
            for comp, loss in (("dot", "ranking"), ("dot", "logistic"), ("l2", "softmax"))])


@pytest.mark.parametrize("test,args,tier", [pytest.param(test, args, tier, id=f"{name}-{tier}") for name, test, args, tier in SMALL])
def test_separate_kernels_on_small_shapes(test, args, tier, monkeypatch):
    """The same for the other tests whose shapes the one-kernel path takes by default."""
    monkeypatch.setenv("PBG_CHUNK", "0")
    with steps._tier_tolerance(tier):
        test(*args)


@pytest.mark.parametrize("tier", steps.PLANE_TIERS)
def test_fused_kernels_with_global_embeddings(tier, monkeypatch):
    """Waves of several batches with global vectors through the fused score + loss kernel and the dual gradient."""
    monkeypatch.setenv("PBG_CHUNK", "0")
    monkeypatch.setenv("PBG_FUSED", "1")
    with steps._tier_tolerance(tier):
        steps.test_wave_with_global_embeddings_matches_oracle(tier)
