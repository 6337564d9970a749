"""The device RankingEvaluator against ranks / MRR / hits computed from the oracle's forward scores
(eval.py:43-81 restated in NumPy here: rank = 1 + #(neg >= pos), both sides averaged)."""
import numpy as np
import pytest

from golden_util import batch_of, load_step, oracle_config, oracle_state
from oracle import pbg_step as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["partial_last_chunk", "c3_none_dot_softmax", "c5_dyn_complex_l2_logistic",
                                  "std_linear_dot_ranking", "disable_lhs_negs", "uniform_only_mode"])
def test_ranking_evaluator_matches_oracle_scores(name):
    import torchbiggraph_b200 as T
    from b200_util import Rig
    c, z = load_step(name)
    ocfg, ost = oracle_config(c), oracle_state(c, z)
    rig = Rig.from_oracle_state(c, ost)
    lhs, rhs, rel, ul, ur = batch_of(c, z, 0)
    sc = O.score_batch(ocfg, ost, lhs, rhs, rel, ul, ur)
    ev = T.B200RankingEvaluator(T.LOSS_FUNCTIONS.get_class(c["loss"])(margin=c["margin"]),
                                [r.weight for r in rig.cfg.relations])
    st = ev.process_one_batch(rig.model, rig.edges(lhs, rhs, rel), ul, ur)
    n = len(lhs)
    ranks, aucs, losses = [], [], 0.0
    for side in ("lhs", "rhs"):
        pos, neg = sc[f"{side}_pos"], sc[f"{side}_neg"]
        val, _, _ = O.loss_forward_backward(c["loss"], c["margin"], pos, neg)
        losses += val
        if neg.size:
            ranks.append((neg >= pos[:, None]).sum(1) + 1)
            aucs.append(float((pos[:, None] > neg).mean()))      # exact value the randomized AUC estimates
    w = 1.0 if c["dyn"] else ([c["rel_weight"] if i == c["rel_idx"] else 1.0 for i in range(c["n_rel_std"])][c["rel_idx"]])
    assert st.count == n
    assert st.metrics["loss"] == pytest.approx(w * losses, rel=1e-4, abs=1e-3)
    mean_of_sums = lambda xs: float(np.mean([x.sum() for x in xs]))
    # a negative that ties with its positive (same entity) may fall either side of `>=` in fp32
    ties = sum(int((np.abs(sc[f"{s}_neg"] - sc[f"{s}_pos"][:, None]) <= 2e-5 * (1 + np.abs(sc[f"{s}_pos"][:, None]))).sum())
               for s in ("lhs", "rhs"))
    assert abs(st.metrics["pos_rank"] - mean_of_sums(ranks)) <= ties / len(ranks) + 1e-6
    assert abs(st.metrics["mrr"] - mean_of_sums([1.0 / r for r in ranks])) <= ties / len(ranks) + 1e-4
    for key, lim in (("r1", 1), ("r10", 10), ("r50", 50)):
        assert abs(st.metrics[key] - mean_of_sums([(r <= lim) for r in ranks])) <= ties / len(ranks) + 1e-6
    # `count` random pairs per side: standard error of the mean AUC is at most 0.5 / sqrt(count)
    assert abs(st.metrics["auc"] / n - float(np.mean(aucs))) <= 4 * 0.5 / np.sqrt(n)


def _mix64(z):
    """The kernels' hash (splitmix64's finalizer)."""
    m = 2**64 - 1
    z = z + 0x9E3779B97F4A7C15 & m
    z = (z ^ z >> 30) * 0xBF58476D1CE4E5B9 & m
    z = (z ^ z >> 27) * 0x94D049BB133111EB & m
    return z ^ z >> 31


def _auc_samples(seed, side, count, cols, all_negs=False):
    """The (positive, edge of the negative, its column) triples that the evaluator draws on one side."""
    for i in range(count):
        h = _mix64(seed ^ _mix64((0xA11CE5 if all_negs else 0xA0C0FFEE) + side * 0x10001 + i))
        e, h = h % count, _mix64(h)
        if all_negs:
            yield e, h % count, _mix64(h) % cols
        else:
            yield e, h % (count * cols) // cols, h % (count * cols) % cols


def _allnegs_rig(z, cfg_o, st_o):
    """Model and evaluator for a recorded all_negs case (tests/golden/allnegs_*.npz)."""
    import torch
    import torchbiggraph_b200 as T
    sep, dyn = bool(z["separate"]), bool(z["dyn"])
    ents = {"e": T.EntitySchema()}
    rhs_ent = "e"
    if sep:
        ents["f"] = T.EntitySchema()
        rhs_ent = "f"
    cfg = T.ConfigSchema(entities=ents, relations=[T.RelationSchema("r0", "e", rhs_ent, operator=str(z["op"]), all_negs=True)],
                         dimension=z["W_lhs"].shape[1], comparator=str(z["comp"]), loss_fn=str(z["loss"]), margin=float(z["margin"]),
                         batch_size=1000, num_batch_negs=50, num_uniform_negs=0, dynamic_relations=dyn,
                         num_dynamic_rels=int(z["R"]) if dyn else 0)
    model = T.make_model(cfg, "cuda")
    f32 = lambda a: torch.tensor(np.asarray(a, np.float32), device="cuda").contiguous()
    Wl = f32(z["W_lhs"])
    Wr = f32(z["W_rhs"]) if sep else Wl
    model.set_embeddings("e", T.Side.LHS, Wl)
    model.set_embeddings(rhs_ent, T.Side.RHS, Wr)
    if model.rhs_op_table is not None:
        model.rhs_op_table.copy_(f32(z["theta_rhs"]))
    if model.lhs_op_table is not None:
        model.lhs_op_table.copy_(f32(z["theta_lhs"]))
    ev = T.B200RankingEvaluator(T.LOSS_FUNCTIONS.get_class(str(z["loss"]))(margin=float(z["margin"])), [1.0])
    return T, model, ev


def _allnegs_names():
    from test_oracle_golden import allnegs_cases
    return allnegs_cases()


@pytest.mark.parametrize("name", _allnegs_names())
def test_ranking_against_all_entities_matches_the_reference_evaluator(name):
    """Relations with all_negs=True: rank of the true entity among ALL rows of the side's table, the true entity itself
    ignored (model.py:582-617), against the Stats the reference's RankingEvaluator returned for the same batch."""
    import torch
    from test_oracle_golden import allnegs_stats, load_allnegs
    cfg_o, st_o, z = load_allnegs(name)
    T, model, ev = _allnegs_rig(z, cfg_o, st_o)
    t = lambda a: torch.tensor(np.asarray(a, np.int64))
    edges = T.EdgeList(T.EntityList.from_tensor(t(z["lhs"])), T.EntityList.from_tensor(t(z["rhs"])), t(z["rel"]))
    st = ev.process_one_batch(model, edges)
    n = int(z["stat_count"])
    assert st.count == n
    assert st.metrics["loss"] == pytest.approx(float(z["stat_loss"]), rel=1e-4)
    # candidates whose score ties with the positive up to fp32 rounding may fall either side of `>=`
    sc = O.score_all_negs(cfg_o, st_o, z["lhs"], z["rhs"], z["rel"])
    ties = sum(int((np.abs(sc[f"{s}_neg"] - sc[f"{s}_pos"][:, None]) <= 2e-5 * (1 + np.abs(sc[f"{s}_pos"][:, None]))).sum()) for s in ("lhs", "rhs"))
    assert abs(st.metrics["pos_rank"] - float(z["stat_pos_rank"])) <= ties / 2 + 1e-6
    assert abs(st.metrics["mrr"] - float(z["stat_mrr"])) <= ties / 2 + 1e-4
    for k in ("r1", "r10", "r50"):
        assert abs(st.metrics[k] - float(z["stat_" + k])) <= ties / 2 + 1e-6
    exact_auc = allnegs_stats(cfg_o, sc)["auc"]
    assert abs(st.metrics["auc"] / n - exact_auc) <= 4 * 0.5 / np.sqrt(n)
    # ... and sample by sample; of those that tie as above either outcome will do
    hits = unsure = 0
    for side, (pos, neg) in enumerate(((sc["lhs_pos"], sc["lhs_neg"]), (sc["rhs_pos"], sc["rhs_neg"]))):
        for e, er, j in _auc_samples(ev.seed + ev._calls, side, n, neg.shape[1], all_negs=True):
            hits += pos[e] > neg[er, j]
            unsure += abs(pos[e] - neg[er, j]) <= 2e-5 * (1 + abs(pos[e]))
    assert abs(2 * st.metrics["auc"] - hits) <= unsure


def test_all_negs_relations_are_not_trained():
    from test_oracle_golden import load_allnegs
    import torch
    cfg_o, st_o, z = load_allnegs("std_translation_dot_softmax")
    T, model, ev = _allnegs_rig(z, cfg_o, st_o)
    tr = T.B200Trainer(T.make_optimizer(model.config, model.parameters(), False), T.LOSS_FUNCTIONS.get_class("softmax")(margin=0.1), [1.0])
    tr.partitioned_optimizers["e", 0] = T.make_optimizer(model.config, [model.lhs_embs["emb_e"]], True)
    t = lambda a: torch.tensor(np.asarray(a, np.int64))
    with pytest.raises(NotImplementedError, match="all_negs"):
        tr.process_one_batch(model, T.EdgeList(T.EntityList.from_tensor(t(z["lhs"])), T.EntityList.from_tensor(t(z["rhs"])), t(0)))


@pytest.mark.parametrize("loss", ["softmax", "ranking", "logistic"])
@pytest.mark.parametrize("B,nb,nu", [(1, 1, 3), (23, 7, 3), (130, 130, 390), (513, 513, 0), (515, 128, 2), (70, 0, 35)])
def test_sampled_ranks_are_the_ranks_of_the_forward_scores(B, nb, nu, loss, monkeypatch):
    """Rows whose own column lies at every place of a group of four, chunks that end inside one, more columns than one pass of a
    warp takes, no batch negatives, samples of the AUC that end inside a CTA of 256: ranks, hits and samples are counts over the
    scores that the forward call returns for the same candidates (PBG_CHUNK=0: by the evaluator's own kernels, so they are equal),
    the loss is its formula in double precision over those scores.  The device
    adds up to 520 terms in single precision: 520 x 2^-24 = 3.1e-5 relative, and the terms' own rounding (exp, log: a few 2^-24)."""
    import torch
    import torchbiggraph_b200 as T
    monkeypatch.setenv("PBG_CHUNK", "0")
    g = torch.Generator().manual_seed(B + nb)
    rows, D, margin, chunks = 900, 20, 0.1, -(-B // (nb or nu))
    cfg = T.ConfigSchema(entities={"e": T.EntitySchema()}, relations=[T.RelationSchema("r", "e", "e", operator="none")], dimension=D,
                         comparator="dot", loss_fn=loss, margin=margin, batch_size=chunks * (nb or nu), num_batch_negs=nb, num_uniform_negs=nu, precision="fp32")
    m = T.make_model(cfg, "cuda")
    W = torch.randn(rows, D, generator=g).cuda()
    m.set_embeddings("e", T.Side.LHS, W)
    m.set_embeddings("e", T.Side.RHS, W)
    edges = T.EdgeList(T.EntityList.from_tensor(torch.randint(0, rows, (B,), generator=g)), T.EntityList.from_tensor(torch.randint(0, rows, (B,), generator=g)), torch.tensor(0))
    ul, ur = (torch.randint(0, rows, (chunks, nu), generator=g).cuda() if nu else None for _ in range(2))
    sc = m(edges, ul, ur)
    ev = T.B200RankingEvaluator(T.LOSS_FUNCTIONS.get_class(loss)(margin=margin), [1.0])
    st = ev.process_one_batch(m, edges, ul, ur)
    want, value = np.zeros(6), 0.0
    for side, (pos, neg) in enumerate(((sc.lhs_pos, sc.lhs_neg), (sc.rhs_pos, sc.rhs_neg))):
        pos, neg = pos.double().cpu(), neg.double().cpu()
        rk = 1 + (neg >= pos[:, None]).sum(1)
        hits = sum(bool(pos[e] > neg[er, j]) for e, er, j in _auc_samples(ev.seed + ev._calls, side, B, neg.shape[1]))
        want += [x / 2 for x in (float(rk.sum()), *(float((rk <= k).sum()) for k in (1, 10, 50)), float((1.0 / rk.double()).sum()), hits)]
        if loss == "softmax":
            value += float((torch.logsumexp(torch.cat([pos[:, None], neg], 1), 1) - pos).sum())
        elif loss == "ranking":
            value += float((neg - pos[:, None] + margin).clamp(min=0).sum())
        else:
            sp = torch.nn.functional.softplus
            value += float(sp(-pos).sum() + sp(neg).sum() / neg.shape[1])
    assert [st.metrics[k] for k in ("pos_rank", "r1", "r10", "r50", "mrr", "auc")] == pytest.approx(list(want), abs=1e-9)
    assert st.metrics["loss"] == pytest.approx(value, rel=4e-5, abs=1e-5)
