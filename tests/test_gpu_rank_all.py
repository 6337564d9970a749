"""Ranking against all entities at the edges of its tiles: one edge and one more than a tile of 128, tables just below, at and
above a tile of 256 candidates and beyond one slab, dimensions off the 32-value blocks -- tensor-core tiers and the fp32
tier against each other (ranks are integers: they agree except where rounding decides a near tie) and the oracle's ranks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stats(rows, D, B, comp, loss, precision, seed=3, **options):
    import torchbiggraph_b200 as T
    g = torch.Generator().manual_seed(seed)
    cfg = T.ConfigSchema(entities={"e": T.EntitySchema()}, relations=[T.RelationSchema("r", "e", "e", operator="translation", all_negs=True)],
                         dimension=D, comparator=comp, loss_fn=loss, batch_size=200, num_batch_negs=50, num_uniform_negs=50, precision=precision, **options)
    m = T.make_model(cfg, "cuda")
    W = (torch.randn(rows, D, generator=g) * D ** -0.5)
    t = torch.randn(1, D, generator=g) * 0.3 * D ** -0.5
    m.rhs_op_table.copy_(t)
    Wc = W.cuda()
    m.set_embeddings("e", T.Side.LHS, Wc)
    m.set_embeddings("e", T.Side.RHS, Wc)
    lhs, rhs = (torch.randint(0, rows, (B,), generator=g) for _ in range(2))
    ev = T.B200RankingEvaluator(T.LOSS_FUNCTIONS.get_class(loss)(margin=0.1), [1.0])
    s = ev.process_one_batch(m, T.EdgeList(T.EntityList.from_tensor(lhs), T.EntityList.from_tensor(rhs), torch.tensor(0)))
    return s, W.double(), t.double(), lhs, rhs


@pytest.mark.parametrize("rows,D,B", [(40, 4, 1), (255, 36, 128), (256, 64, 129), (257, 100, 77), (9000, 52, 130), (70_000, 16, 33)])
@pytest.mark.parametrize("comp,loss", [("dot", "softmax"), ("cos", "ranking"), ("l2", "logistic")])
def test_ranks_agree_with_double_precision(rows, D, B, comp, loss):
    got = {p: _stats(rows, D, B, comp, loss, p) for p in ("fp32", "tf32x3", "bf16x3")}
    _, W, t, lhs, rhs = got["fp32"]
    X, Y = W, W + t
    if comp == "cos":
        X, Y = X / X.norm(dim=1, keepdim=True), Y / Y.norm(dim=1, keepdim=True)

    def scores(a, b):
        return a @ b.T if comp != "l2" else -torch.cdist(a, b)
    total = 0.0
    for q, cand, true in ((Y[rhs], X, lhs), (X[lhs], Y, rhs)):
        S = scores(q, cand)
        pos = S[torch.arange(B), true].clone()
        S[torch.arange(B), true] = -float("inf")
        total += float((1 + (S >= pos[:, None]).sum(1)).sum())
    for p, (s, *_) in got.items():
        assert abs(s.metrics["pos_rank"] - total / 2) <= max(1.0, 2e-4 * total), (p, s.metrics["pos_rank"], total / 2)
        np.testing.assert_allclose(s.metrics["loss"], got["fp32"][0].metrics["loss"], rtol=2e-5)
        assert abs(s.metrics["auc"] - got["fp32"][0].metrics["auc"]) <= 1.0


@pytest.mark.parametrize("precision", ["fp32", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("off", [("lhs",), ("rhs",), ("lhs", "rhs")], ids="+".join)
def test_sides_without_negatives_count_for_nothing(precision, off):
    """Neither side: no candidates, so no slab and no score tile is launched, and every sum is zero.  One side: the averages of the
    evaluator are the other side's."""
    options = {f"disable_{side}_negs": True for side in off}
    s, W, t, lhs, rhs = _stats(300, 36, 70, "dot", "softmax", precision, **options)
    assert s.count == 70
    if len(off) == 2:
        assert all(s.metrics[m] == 0 for m in ("loss", "pos_rank", "mrr", "r1", "r10", "r50", "auc"))
        return
    X, Y = W, W + t
    S, true = (Y[rhs] @ X.T, lhs) if off == ("rhs",) else (X[lhs] @ Y.T, rhs)
    i = torch.arange(70)
    pos = S[i, true].clone()
    np.testing.assert_allclose(s.metrics["loss"], float((torch.logsumexp(S, 1) - pos).sum()), rtol=1e-5)
    S[i, true] = -float("inf")
    total = float((1 + (S >= pos[:, None]).sum(1)).sum())
    assert abs(s.metrics["pos_rank"] - total) <= 1.0
