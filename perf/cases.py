"""The calls that a user of torchbiggraph_b200 makes, as measurable cases.

A case is one call (or one short sequence of calls) through the package's public entry points, on tables and edge
lists of a stated size:

  kind "batch"      B200Trainer.process_one_batch: one batch, the unit the reference's trainer works in
  kind "train"      process_in_batches: a bucket's whole edge list, batch after batch
  kind "eval"       B200RankingEvaluator.process_one_batch against sampled negatives
  kind "eval_all"   the same for a relation with all_negs: every entity of a side is a negative
  kind "score"      MultiRelationEmbedder.forward against sampled candidates only
  kind "edges"      the edge-list utilities a bucket goes through before it is trained (randperm, sub_bucket) and
                    after an epoch (reverse_permutation, shuffle)

Tables hold what they hold in the middle of a training run: scores of order one, accumulators that have seen a few
hundred steps.  Endpoints follow a power law over randomly permuted ids (`skew` is the exponent over ranks, 0 =
uniform), relations a Zipf law.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "pytorch-biggraph_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import torchbiggraph_b200 as T  # noqa: E402
from torchbiggraph_b200 import _C as edge_utils  # noqa: E402

DEVICE = "cuda"


def _model_case(name, kind, **kw):
    case = dict(name=name, kind=kind, dim=100, op="none", comp="cos", loss="ranking", dynamic=False, rels=1, rel_zipf=1.0,
                rows_lhs=100_000, rows_rhs=100_000, shared=False, skew=1.0, batch=1000, nb=50, nu=50, k=1, precision="fp32",
                edges=1000, host_edges=False, weighted=False, global_emb=False, reg=0.0, max_norm=0.0)
    unknown = set(kw) - set(case)
    assert not unknown, unknown
    case.update(kw)
    return case


def listed():
    return [
        # the smallest call in earnest: a hand-fed batch with per-edge weights whose sizes fit nothing (37 edges, chunks of 15)
        _model_case("one_batch_ragged", "batch", dim=52, op="diagonal", comp="l2", loss="logistic", rows_lhs=5_003, rows_rhs=7_919,
                    skew=0.75, batch=45, nb=15, nu=7, precision="tf32x3", edges=37, weighted=True),
        # one batch under the configuration defaults (cos, ranking, 1000 edges, 50 + 50 negatives, fp32, sequential)
        _model_case("one_batch_default", "batch", shared=True, skew=1.1),
        # scoring edges against uniformly sampled candidates, no update
        _model_case("score_candidates", "score", dim=200, op="translation", comp="cos", rows_lhs=200_000, rows_rhs=150_001, nb=0, nu=100,
                    precision="tf32x3"),
        # held-out evaluation of a multi-relation graph of 15k entities: 5000 edges against 1000 batch negatives a side
        _model_case("eval_sampled", "eval", dim=400, op="complex_diagonal", comp="dot", loss="softmax", dynamic=True, rels=1345,
                    rows_lhs=14_951, rows_rhs=14_951, shared=True, skew=0.0, batch=5000, nb=1000, nu=0, precision="tf32x3", edges=5000),
        # full ranking: the same graph, every entity a negative
        _model_case("eval_all_entities", "eval_all", dim=400, op="translation", comp="cos", loss="softmax", rows_lhs=14_951,
                    rows_rhs=14_951, shared=True, skew=0.0, batch=1000, nb=50, nu=50, precision="tf32x3"),
        # a bucket's edges on their way to training: shuffle, split into 2 x 2 sub-partitions; table rows permuted and back
        dict(name="edge_list_utilities", kind="edges", edges=269_507, rows_lhs=302_974, rows_rhs=302_973, dim=100, rels=1, parts_lhs=2,
             parts_rhs=2),
        # sequential semantics (one batch in flight) over twelve relations of one entity type, with the global embedding that
        # is the reference's default; edges in pinned host memory, as the reference's reader leaves them
        _model_case("bucket_sequential", "train", dim=128, op="translation", comp="cos", loss="softmax", rels=12, rows_lhs=120_000,
                    rows_rhs=120_000, skew=0.8, precision="tf32x3", edges=49_950, host_edges=True, global_emb=True),
        # the plumbing graph: one table, dimension 100, a million edges, fourteen batches in flight
        _model_case("bucket_plumbing", "train", op="none", comp="dot", loss="ranking", shared=True, skew=1.1, k=14,
                    precision="bf16x6", edges=1_000_000),
        # a bucket of a follower graph: two partitions of 2.6 million rows, translation / cos, two-plane tier
        _model_case("bucket_follower", "train", op="translation", comp="cos", loss="ranking", rows_lhs=2_603_265, rows_rhs=2_603_264,
                    skew=1.0, nb=100, nu=100, k=14, precision="bf16x3", edges=269_507, host_edges=True),
        # a bucket of a large knowledge graph: 14,824 relations with operators of their own, logistic loss on l2 distances
        _model_case("bucket_knowledge", "train", dim=200, op="complex_diagonal", comp="l2", loss="logistic", dynamic=True, rels=14_824,
                    rel_zipf=1.2, rows_lhs=5_378_379, rows_rhs=5_378_378, skew=0.0, nb=100, nu=100, k=14, precision="tf32x3",
                    edges=269_507),
        # a bucket of the social graph: dimension 1024, softmax on dot products
        _model_case("bucket_social", "train", dim=1024, op="none", comp="dot", loss="softmax", rows_lhs=302_974, rows_rhs=302_973,
                    skew=0.77, nb=100, nu=100, k=14, precision="bf16x6", edges=269_507),
        # one pass over the 15k-entity multi-relation graph: batches of 5000 with 1000 batch negatives, three in flight
        _model_case("bucket_small_graph", "train", dim=400, op="complex_diagonal", comp="dot", loss="softmax", dynamic=True, rels=1345,
                    rows_lhs=14_951, rows_rhs=14_951, shared=True, skew=0.0, batch=5000, nb=1000, nu=0, k=3, precision="tf32x3",
                    edges=483_142),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "train", "train", "train", "train", "train", "eval", "eval_all", "score", "edges"])
    if kind == "edges":
        return dict(kind=kind, edges=_log_int(rng, 1_000, 269_507), rows_lhs=_log_int(rng, 1_000, 300_000),
                    rows_rhs=_log_int(rng, 1_000, 300_000), dim=rng.choice([4, 25, 50, 100, 101, 256]), rels=rng.choice([1, 1, 3, 12]),
                    parts_lhs=rng.randint(1, 4), parts_rhs=rng.randint(1, 4))
    dynamic = kind != "eval_all" and rng.random() < 0.35
    op = rng.choice(["complex_diagonal", "diagonal", "translation"] if dynamic else ["none", "none", "diagonal", "translation", "complex_diagonal"])
    dim = 8 * _log_int(rng, 2, 128) if op == "complex_diagonal" else 4 * _log_int(rng, 4, 256)
    big_chunks = dynamic and dim <= 400 and rng.random() < 0.3
    nb = _log_int(rng, 250, 1000) if big_chunks else _log_int(rng, 10, 120)
    nu = 0 if big_chunks else _log_int(rng, 5, 120)
    chunks = rng.randint(2, 5) if big_chunks else rng.randint(4, 20)
    if kind == "score":
        nb, nu, chunks = 0, _log_int(rng, 10, 120), rng.randint(4, 20)
    batch = (nb or nu) * chunks
    k = 1 if kind != "train" else rng.choice([1, 2, 4] if big_chunks else [1, 4, 8, 14, 14])
    many = kind == "train" and not dynamic and rng.random() < 0.3
    comp = rng.choice(["dot", "cos", "l2"])
    # an edge of a wide model costs more: the list gets shorter with the dimension, so that no draw outweighs the listed cases
    most = max(4 * batch, min(269_507, int(2.0e7 / dim) if k > 1 else int(3.0e6 / dim)))
    edges = _log_int(rng, 2 * batch, most) if kind == "train" else rng.randint(max(1, batch // 3), batch)
    rows_lhs = _log_int(rng, 5_000, 20_000) if kind == "eval_all" else _log_int(rng, 50_000 if kind == "eval" else 5_000, 1_000_000)
    shared = rng.random() < 0.3
    case = _model_case("", kind, dim=dim, op=op, comp=comp, loss=rng.choice(["softmax", "ranking", "logistic"]), dynamic=dynamic,
                       rels=_log_int(rng, 10, 15_000) if dynamic else (rng.randint(2, 12) if many else 1),
                       rel_zipf=rng.choice([1.0, 1.2]), rows_lhs=rows_lhs, rows_rhs=rows_lhs if shared else _log_int(rng, min(rows_lhs, 50_000 if kind == "eval" else 5_000), rows_lhs),
                       shared=shared, skew=0.0 if kind == "eval" else rng.choice([0.0, 0.77, 1.0]), batch=batch, nb=nb, nu=nu, k=k,
                       precision=rng.choice(["fp32", "tf32x3"] if kind in ("batch", "score") else ["tf32x3", "bf16x6", "bf16x6", "bf16x3"]),
                       edges=edges, host_edges=kind == "train" and rng.random() < 0.5, weighted=kind in ("batch", "train") and rng.random() < 0.2,
                       global_emb=not dynamic and rng.random() < 0.15)
    if kind in ("batch", "train") and rng.random() < 0.1:
        case["reg"] = 1e-3
    if kind in ("batch", "train") and rng.random() < 0.1:
        case["max_norm"] = 1.0
    del case["name"]
    return case


# ---- inputs --------------------------------------------------------------------------------------------------------
def _power_law(n, rows, skew, gen):
    """`n` row ids, the i-th most popular of `rows` with probability proportional to (i + 1) ** -skew, ids permuted."""
    if skew == 0.0:
        return torch.randint(0, rows, (n,), device=DEVICE, generator=gen)
    cdf = torch.arange(1, rows + 1, device=DEVICE, dtype=torch.float64).pow_(-skew).cumsum_(0)
    rank = torch.searchsorted(cdf, torch.rand(n, device=DEVICE, generator=gen, dtype=torch.float64) * cdf[-1]).clamp_(max=rows - 1)
    return torch.randperm(rows, device=DEVICE, generator=gen)[rank]


def _scale(case):
    """Size of a table entry: scores are of order one."""
    return case["dim"] ** (-0.25 if case["comp"] == "dot" else -0.5)


def _sums(shape, visits, case, gen):
    """Adagrad sums after `visits` gradients.  A positive pulls its row once (softmax, logistic) or once per negative
    inside the margin (ranking, about half of them)."""
    pull = 0.5 * (case["nb"] + case["nu"]) if case["loss"] == "ranking" else 1.0
    return torch.rand(shape, device=DEVICE, generator=gen).add_(0.5).mul_(visits * (pull * _scale(case)) ** 2)


def _table(rows, case, gen):
    """A partition in the middle of a training run: its rows and their RowAdagrad sums."""
    return torch.randn(rows, case["dim"], device=DEVICE, generator=gen).mul_(_scale(case)), _sums((rows,), 100, case, gen)


def _prepare_edges_case(case, gen):
    n = case["edges"]
    return dict(case=case, seed=int(torch.randint(0, 1 << 30, (1,), device=DEVICE, generator=gen)),
                lhs=torch.randint(0, case["rows_lhs"], (n,), device=DEVICE, generator=gen),
                rhs=torch.randint(0, case["rows_rhs"], (n,), device=DEVICE, generator=gen),
                rel=torch.randint(0, case["rels"], (n,), device=DEVICE, generator=gen),
                perm_lhs=torch.randperm(case["rows_lhs"], device=DEVICE, generator=gen),
                perm_rhs=torch.randperm(case["rows_rhs"], device=DEVICE, generator=gen),
                table=torch.randn(case["rows_lhs"], case["dim"], device=DEVICE, generator=gen),
                out=[torch.empty(n, dtype=torch.long, device=DEVICE) for _ in range(3)])


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    if case["kind"] == "edges":
        return _prepare_edges_case(case, gen)
    dyn, rels = case["dynamic"], case["rels"]
    schema = [T.RelationSchema("r%d" % i, "e", "e", operator=case["op"], all_negs=case["kind"] == "eval_all")
              for i in range(1 if dyn else rels)]
    cfg = T.ConfigSchema(entities={"e": T.EntitySchema(num_partitions=1 if case["shared"] else 2)}, relations=schema, dimension=case["dim"],
                         comparator=case["comp"], loss_fn=case["loss"], margin=0.1, lr=0.1, batch_size=case["batch"],
                         num_batch_negs=case["nb"], num_uniform_negs=case["nu"], dynamic_relations=dyn,
                         num_dynamic_rels=rels if dyn else 0, precision=case["precision"], batches_in_flight=case["k"],
                         global_emb=case["global_emb"], regularization_coef=case["reg"], max_norm=case["max_norm"] or None)
    model = T.make_model(cfg, DEVICE)
    model_optimizer = T.make_optimizer(cfg, model.parameters(), False)
    for p in model.parameters():                                       # operators and global vectors away from their initial values
        step = _scale(case) if case["op"] == "translation" or p.dim() == 1 else 1.0
        p.add_(torch.randn(p.shape, device=DEVICE, generator=gen), alpha=0.1 * step)
        model_optimizer.sum_for(p).copy_(_sums(p.shape, 100.0 * max(1.0, case["batch"] / rels), case, gen))
    loss_fn = T.LOSS_FUNCTIONS.get_class(case["loss"])(margin=0.1)
    weights = [1.0] * len(schema)
    state = dict(case=case, model=model, seed=seed, tables={})
    lhs_w, lhs_sum = _table(case["rows_lhs"], case, gen)
    rhs_w, rhs_sum = (lhs_w, lhs_sum) if case["shared"] else _table(case["rows_rhs"], case, gen)
    model.set_embeddings("e", T.Side.LHS, lhs_w)
    model.set_embeddings("e", T.Side.RHS, rhs_w)
    if case["kind"] in ("batch", "train"):
        trainer = T.B200Trainer(model_optimizer, loss_fn, weights)
        for part, (side, w, s) in enumerate([("lhs", lhs_w, lhs_sum), ("rhs", rhs_w, rhs_sum)][:1 if case["shared"] else 2]):
            opt = T.RowAdagrad([w], lr=cfg.lr)
            opt.sum_for(w).copy_(s)
            trainer.partitioned_optimizers["e", part] = opt
            state["tables"][side] = w
            state["tables"][side + "_sum"] = opt.sum_for(w)
        for i, p in enumerate(model.parameters()):
            state["tables"]["param%d" % i] = p
            state["tables"]["param%d_sum" % i] = model_optimizer.sum_for(p)
        state["trainer"] = trainer
    elif case["kind"] in ("eval", "eval_all"):
        state["evaluator"] = T.B200RankingEvaluator(loss_fn, weights)
    n = case["edges"]
    lhs = _power_law(n, case["rows_lhs"], case["skew"], gen)
    rhs = _power_law(n, case["rows_rhs"], case["skew"], gen)
    rel = torch.tensor(0)
    if rels > 1:
        law = torch.arange(1, rels + 1, device=DEVICE, dtype=torch.float64).pow_(-case["rel_zipf"]).cumsum_(0)
        rel = torch.searchsorted(law, torch.rand(n, device=DEVICE, generator=gen, dtype=torch.float64) * law[-1]).clamp_(max=rels - 1)
        if not dyn and case["kind"] != "train":
            rel = rel[0].cpu()                                         # a single batch holds one relation
    weight = torch.rand(n, device=DEVICE, generator=gen).add_(0.5) if case["weighted"] else None
    if case["host_edges"]:
        lhs, rhs = lhs.cpu().pin_memory(), rhs.cpu().pin_memory()
        rel = rel.cpu().pin_memory() if rel.dim() else rel
        weight = weight.cpu().pin_memory() if weight is not None else None
    state["edges"] = T.EdgeList(T.EntityList.from_tensor(lhs), T.EntityList.from_tensor(rhs), rel, weight)
    return state


# ---- the calls -----------------------------------------------------------------------------------------------------
def _stats(s):
    """Stats as outputs.  The training loss's companion counts, the violators, are read but not returned: a batch
    negative that is the edge's own entity ties with the positive, rounding decides which is larger, and on a power-law
    graph those ties are a tenth of the count."""
    out = {"count": s.count, "loss": float(s.metrics["loss"] + s.metrics.get("reg", 0.0))}
    if "pos_rank" in s.metrics:
        out["ranks"] = torch.tensor([s.metrics[c] for c in ("pos_rank", "mrr", "r1", "r10", "r50", "auc")], dtype=torch.float64)
    return out


def _run_edges_case(st):
    case = st["case"]
    order = edge_utils.randperm(case["edges"], seed=st["seed"])
    lhs, rhs, rel = st["lhs"][order], st["rhs"][order], st["rel"][order]
    rels = case["rels"]
    parts = edge_utils.sub_bucket(lhs, rhs, rel, [case["rows_lhs"]] * rels, [st["perm_lhs"]] * rels, [case["rows_rhs"]] * rels,
                                  [st["perm_rhs"]] * rels, *st["out"], case["parts_lhs"], case["parts_rhs"])
    back = edge_utils.reverse_permutation(st["perm_lhs"])
    edge_utils.shuffle(st["table"], st["perm_lhs"])
    return {"order": order, "sizes": [p[0].shape[0] for p in parts.values()], "edges": st["out"], "back": back, "table": st["table"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "edges":
        return _run_edges_case(state)
    model, edges = state["model"], state["edges"]
    if kind == "train":
        torch.default_generator.manual_seed(state["seed"])            # the order in which relations take turns is drawn on the host
        stats = T.process_in_batches(case["batch"], model, state["trainer"], edges)
        return {"stats": _stats(stats), "state": state["tables"]}
    if kind == "batch":
        return {"stats": _stats(state["trainer"].process_one_batch(model, edges)), "state": state["tables"]}
    if kind == "score":
        return list(model.forward(edges, seed=state["seed"]))
    return _stats(state["evaluator"].process_one_batch(model, edges))


# ---- what a call cannot do without ---------------------------------------------------------------------------------
def work(case):
    """Bytes: every input read once and every output written once.  A trained edge touches two rows and its share of
    the uniform negatives on both sides, each read in the forward pass, and read and written by the optimizer."""
    n, D = case["edges"], case["dim"]
    if case["kind"] == "edges":
        perms = case["rows_lhs"] + case["rows_rhs"]
        return {"bytes": 8.0 * (n + 6 * n + 3 * n + perms + 2 * case["rows_lhs"]) + 8.0 * D * case["rows_lhs"], "flops": 0.0}
    if case["kind"] == "eval_all":
        rows = case["rows_lhs"] + (0 if case["shared"] else case["rows_rhs"])
        return {"bytes": 4.0 * D * (rows + 2 * n) + 16.0 * n, "flops": 2.0 * D * n * (case["rows_lhs"] + case["rows_rhs"])}
    P, U = case["nb"] or case["nu"], case["nu"]
    P = min(P, n)
    cols = (P if case["nb"] else 0) + U
    rows = 2.0 * n + 2.0 * U * math.ceil(n / P)                        # table rows looked up, duplicates included
    edge_bytes = 24.0 if case["dynamic"] else 16.0
    ops = 2.0 * n if case["dynamic"] and case["op"] != "none" else 0.0   # operator rows looked up
    forward = 4.0 * D * (rows + ops) + edge_bytes * n
    if case["kind"] == "score":
        return {"bytes": forward + 4.0 * 2 * n * (cols + 1), "flops": 4.0 * D * n * cols}
    if case["kind"] == "eval":
        return {"bytes": forward, "flops": 4.0 * D * n * cols}
    return {"bytes": forward + 8.0 * rows * (D + 1) + 16.0 * ops * D, "flops": 12.0 * D * n * cols}


def tolerance(case):
    """How far two correct fp32-accumulating implementations end up apart, from running the cases with the contractions
    in different tiers.  Training amplifies the last bits of a sum through the batches that follow, and the ranking loss
    switches a negative's whole gradient on or off at the margin: a few rows then differ visibly."""
    if case["kind"] == "edges":
        return "exact"
    if case["kind"] == "eval":
        return {"rel": 1e-3, "max": 1e-3}                              # ranks: ties of an entity with itself
    if case["kind"] != "train":
        return {"rel": 1e-5, "max": 3e-4}
    if case["loss"] == "ranking":
        return {"rel": 1e-3, "max": 0.1}
    return {"rel": 3e-4, "max": 1e-2} if case["precision"] == "bf16x3" else {"rel": 1e-4, "max": 5e-3}
