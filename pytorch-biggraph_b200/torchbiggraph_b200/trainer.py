"""The batch processor that replaces the reference's Trainer (torchbiggraph/train_cpu.py:74-112)
and the batch loop around it (torchbiggraph/batching.py:91-125).

`B200Trainer.process_one_batch(model, batch_edges) -> Stats` is the reference interface
(AbstractBatchProcessor, batching.py:128-165).  `process_in_batches` hands a whole edge list to the
library in one call, which trains `batches_in_flight` batches per wave on the device."""
import ctypes as C
import time
import weakref
from abc import ABC, abstractmethod
from typing import Dict, Iterable, List, Optional, Tuple

import numpy as np
import torch

from . import _lib
from ._lib import PbgBatch, PbgBatchStats, PbgBucket, PbgConfig, check
from .model import MultiRelationEmbedder, Scores
from .registries import LOSS_FUNCTIONS, AbstractLossFunction
from .row_adagrad import AsyncAdagrad, RowAdagrad
from .types import EdgeList, Stats


def _ptr(t: Optional[torch.Tensor]):
    return None if t is None else t.data_ptr()


# Device index -> handle of PyTorch's current stream.  (The public form is the same at 3 us a call, which a call of 50 us shows.)
_current_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None) or (lambda index: torch.cuda.current_stream(index).cuda_stream)


# the C structures pbg_batch and pbg_batch_stats as array records
_BATCH = np.dtype([("offset", np.int64), ("count", np.int32), ("rel", np.int32)])
_STATS = np.dtype([("loss", np.float32), ("reg", np.float32), ("violators_lhs", np.int64), ("violators_rhs", np.int64), ("count", np.int64)])


def _even_batches(n: int, batch_size: int, rel: int) -> np.ndarray:
    """Descriptors of n edges of one relation cut into batches of batch_size."""
    out = np.empty(-(-n // batch_size), dtype=_BATCH)
    out["offset"] = np.arange(len(out), dtype=np.int64) * batch_size
    out["count"] = np.minimum(batch_size, n - out["offset"])
    out["rel"] = rel
    return out


class _Native:
    """One library context bound to a model's static configuration."""

    def __init__(self, model: MultiRelationEmbedder, max_batch: int, k: int, precision: str, lr: float,
                 relation_lr: Optional[float], margin: float, loss_code: Optional[int] = None,
                 num_batch_negs: Optional[int] = None, num_uniform_negs: Optional[int] = None,
                 op_name: Optional[str] = None):
        cfg = model.config
        self.op_name = model.operator_name if op_name is None else op_name
        if model.device.type != "cuda":
            raise RuntimeError("torchbiggraph_b200 runs on a CUDA device only (no CPU fallback)")
        self.lib = _lib.lib()
        c = PbgConfig()
        c.dim = cfg.dimension
        c.op = _lib.OPERATOR_CODES[self.op_name]
        c.comparator = model.comparator.native_code
        c.loss = _lib.LOSS_CODES[cfg.loss_fn] if loss_code is None else loss_code
        c.dynamic_relations = int(cfg.dynamic_relations)
        c.num_rels = model.num_dynamic_rels if cfg.dynamic_relations else len(model.op_groups[self.op_name])
        c.num_batch_negs = cfg.num_batch_negs if num_batch_negs is None else num_batch_negs
        c.num_uniform_negs = cfg.num_uniform_negs if num_uniform_negs is None else num_uniform_negs
        c.disable_lhs_negs = int(cfg.disable_lhs_negs)
        c.disable_rhs_negs = int(cfg.disable_rhs_negs)
        c.precision = _lib.PRECISION_CODES[precision]
        c.max_batch_size = max_batch
        c.batches_in_flight = k
        c.margin = margin
        c.lr = lr
        c.relation_lr = lr if relation_lr is None else relation_lr
        c.regularization_coef = float(getattr(cfg, "regularization_coef", 0.0))
        c.max_norm = float(getattr(cfg, "max_norm", None) or 0.0)
        self.cfg = c
        self.max_batch = max_batch
        self.device_index = model.device.index if model.device.index is not None else torch.cuda.current_device()
        self._bucket, self._bucket_key = None, ()
        self.ctx = C.c_void_p()
        self.stream = torch.cuda.current_stream(self.device_index)      # the library's, whatever is current at later calls
        self.stream_handle = self.stream.cuda_stream
        st = self.lib.pbg_create(C.byref(c), self.device_index, C.c_void_p(self.stream_handle), C.byref(self.ctx))
        if st != 0:
            msg = self.lib.pbg_last_error(self.ctx).decode() if self.ctx else ""
            self.lib.pbg_destroy(self.ctx)
            self.ctx = None
            if st == _lib.PBG_ERR_UNSUPPORTED:
                raise NotImplementedError(msg)
            raise _lib.PbgError(st, msg)

    def __del__(self):
        if getattr(self, "ctx", None):
            self.lib.pbg_destroy(self.ctx)
            self.ctx = None

    def ordered(self, fn, *args) -> int:
        """fn(context, *args), in step with the caller's current stream: behind what PyTorch has queued there (the copies
        and index kernels that made the arguments, the last use of memory handed out for outputs) and in front of what it
        queues next (temporaries among the arguments go back to its allocator, tables are read)."""
        if _current_stream(self.device_index) == self.stream_handle:
            return fn(self.ctx, *args)
        current = torch.cuda.current_stream(self.device_index)
        self.stream.wait_stream(current)
        try:
            return fn(self.ctx, *args)
        finally:
            current.wait_stream(self.stream)

    def set_hyper(self, lr, relation_lr, margin):
        check(self.lib.pbg_set_hyperparameters(self.ctx, lr, lr if relation_lr is None else relation_lr, margin), self.ctx)

    def bucket(self, model, relation_idx, states, weights) -> PbgBucket:
        """The call's tables as the library takes them.  `weights`: relation weights of the context's operator group, or
        None.  The structure is kept for as long as every address in it stays the same (filling its fifteen fields
        costs a single-batch call as much as three kernel launches)."""
        wl, wr = model.tables_for(relation_idx)
        rhs_tab, lhs_tab = model.op_table_for(self.op_name)
        glob = model.globals_for(relation_idx)
        tensors = (wl, wr, rhs_tab, lhs_tab) + glob + (() if states is None else states)
        key = (wl.shape[0], wr.shape[0], None if weights is None else tuple(weights)) + tuple([None if t is None else t.data_ptr() for t in tensors])
        if key == self._bucket_key:
            return self._bucket
        b = PbgBucket()
        b.lhs_emb, b.lhs_rows = wl.data_ptr(), wl.shape[0]
        b.rhs_emb, b.rhs_rows = wr.data_ptr(), wr.shape[0]
        if states is not None:
            gl, gr, al, ar = states[:4]
            b.lhs_state, b.rhs_state = gl.data_ptr(), gr.data_ptr()
            b.rhs_op_state = None if ar is None else ar.data_ptr()
            b.lhs_op_state = None if al is None else al.data_ptr()
        b.rhs_op = None if rhs_tab is None else rhs_tab.data_ptr()
        b.lhs_op = None if lhs_tab is None else lhs_tab.data_ptr()
        b.relation_weights = None if weights is None else (C.c_float * len(weights))(*weights)
        gl_, gr_ = glob
        if gl_ is not None:
            b.lhs_global, b.rhs_global = gl_.data_ptr(), gr_.data_ptr()
            if states is not None and len(states) > 4:
                b.lhs_global_state, b.rhs_global_state = states[4].data_ptr(), states[5].data_ptr()
        self._bucket, self._bucket_key = b, key
        return b

    def score(self, model, edges: EdgeList, ul, ur, seed) -> Scores:
        n = len(edges)
        dev = model.device
        lhs = edges.lhs.to_tensor().to(dev).contiguous()
        rhs = edges.rhs.to_tensor().to(dev).contiguous()
        dyn = model.num_dynamic_rels > 0
        if dyn and edges.has_scalar_relation_type():
            raise TypeError("Need relation for each positive pair")
        if not dyn and not edges.has_scalar_relation_type():
            raise TypeError("All positive pairs must come from the same relation")
        rel = edges.rel.to(dev).contiguous() if dyn else None
        relidx = 0 if dyn else edges.get_relation_type_as_scalar()
        local = 0 if dyn else model.group_of[relidx][1]
        # negative columns per side (pbg_neg_columns; model.py:648-656)
        nb, nu = self.cfg.num_batch_negs, self.cfg.num_uniform_negs
        cols = (min(nb, n) if nb > 0 else 0) + nu
        lc, rc = 0 if self.cfg.disable_lhs_negs else cols, 0 if self.cfg.disable_rhs_negs else cols
        lp, rp, ln, rn = torch.empty(n * (2 + lc + rc), device=dev).split((n, n, n * lc, n * rc))
        ln, rn = ln.view(n, lc), rn.view(n, rc)
        ul = None if ul is None else self._uniform(ul, dev)
        ur = None if ur is None else self._uniform(ur, dev)
        b = self.bucket(model, relidx, None, None)
        check(self.ordered(self.lib.pbg_score_batch, C.byref(b), _ptr(lhs), _ptr(rhs), _ptr(rel), n, local,
                           _ptr(ul), _ptr(ur), seed, _ptr(lp), _ptr(rp), _ptr(ln), _ptr(rn)), self.ctx)
        return Scores(lp, rp, ln, rn)

    def _uniform(self, u, dev):
        """[chunks, U] ids of ONE batch -> the library's [1, chunks_per_batch, U] layout."""
        u = torch.as_tensor(u, dtype=torch.long)
        lim = self.cfg.num_batch_negs if self.cfg.num_batch_negs > 0 else self.cfg.num_uniform_negs
        P = min(lim, self.max_batch)
        cm = (self.max_batch + P - 1) // P
        out = torch.zeros((cm, self.cfg.num_uniform_negs), dtype=torch.long)
        out[: u.shape[0]] = u.reshape(u.shape[0], -1).cpu()
        return out.to(dev)

    def chunks_per_batch(self) -> int:
        lim = self.cfg.num_batch_negs if self.cfg.num_batch_negs > 0 else self.cfg.num_uniform_negs
        P = min(lim, self.max_batch)
        return (self.max_batch + P - 1) // P


class AbstractBatchProcessor(ABC):
    """torchbiggraph/batching.py:128-165."""

    def __init__(self, loss_fn: AbstractLossFunction, relation_weights: List[float], overrides=None):
        self.loss_fn = loss_fn
        self.relation_weights = relation_weights
        self.overrides = overrides

    @abstractmethod
    def _process_one_batch(self, model, batch_edges: EdgeList) -> Stats:
        pass

    def process_one_batch(self, model, batch_edges: EdgeList) -> Stats:
        if self.overrides is not None:
            raise NotImplementedError("model overrides are not supported by torchbiggraph_b200")
        return self._process_one_batch(model, batch_edges)


class B200Trainer(AbstractBatchProcessor):
    """Trainer(model_optimizer, loss_fn, relation_weights) of train_cpu.py:74-84.  The coordinator
    fills `partitioned_optimizers[(entity, part)]` / `unpartitioned_optimizers[entity]` with
    RowAdagrad objects on partition swap exactly as it does for the reference."""

    def __init__(self, model_optimizer, loss_fn: AbstractLossFunction, relation_weights: List[float]):
        super().__init__(loss_fn, relation_weights)
        if getattr(loss_fn, "native_code", None) is None:
            raise NotImplementedError(f"loss function {type(loss_fn).__name__} has no device code (no CPU fallback)")
        self.model_optimizer = model_optimizer
        self.unpartitioned_optimizers: Dict[str, RowAdagrad] = {}
        self.partitioned_optimizers: Dict[Tuple, RowAdagrad] = {}
        self._native: Optional[_Native] = None          # the context used last
        self._natives: Dict[str, _Native] = {}          # one per operator group of the model they were made for
        self._native_model = lambda: None               # (a weak reference: an id would be the next model's too)
        self._native_key = None
        self.seed = 0
        self._calls = 0

    # ---- plumbing ------------------------------------------------------------------------------
    def _state_for(self, table: torch.Tensor) -> torch.Tensor:
        ptr = table.data_ptr()
        for opts in (self.partitioned_optimizers, self.unpartitioned_optimizers):
            for opt in opts.values():
                for p in opt.params:
                    if p.data_ptr() == ptr:
                        return opt.sum_for(p)
        raise RuntimeError("no RowAdagrad optimizer registered for an embedding table of this batch")

    def _lr(self) -> float:
        for opt in list(self.partitioned_optimizers.values()) + list(self.unpartitioned_optimizers.values()):
            return opt.lr
        raise RuntimeError("no embedding optimizer registered")

    def _context(self, model: MultiRelationEmbedder, need_batch: int, op_name: Optional[str] = None) -> _Native:
        """The library context of an operator group (one per operator the relations use)."""
        cfg = model.config
        op_name = model.operator_name if op_name is None else op_name
        key = (cfg.batches_in_flight, cfg.precision)
        if self._native_model() is not model or self._native_key != key:
            self._natives = {}
            self._native_model, self._native_key = weakref.ref(model), key
        nat = self._natives.get(op_name)
        if nat is None or nat.max_batch < need_batch:
            margin = getattr(self.loss_fn, "margin", cfg.margin)
            rel_lr = self.model_optimizer.lr if isinstance(self.model_optimizer, AsyncAdagrad) else cfg.relation_lr
            nat = _Native(model, max(cfg.batch_size, need_batch), cfg.batches_in_flight, cfg.precision,
                          self._lr(), rel_lr, margin, loss_code=self.loss_fn.native_code, op_name=op_name)
            self._natives[op_name] = nat
        self._native = nat
        return nat

    def _op_states(self, model, op_name):
        rhs_tab, lhs_tab = model.op_table_for(op_name)
        if rhs_tab is None:
            return None, None
        if not isinstance(self.model_optimizer, AsyncAdagrad):
            raise RuntimeError("the model has operator parameters but model_optimizer is not an AsyncAdagrad over them")
        ar = self.model_optimizer.sum_for(rhs_tab)
        al = None if lhs_tab is None else self.model_optimizer.sum_for(lhs_tab)
        return al, ar

    def train_batches(self, model: MultiRelationEmbedder, lhs: torch.Tensor, rhs: torch.Tensor,
                      rel: Optional[torch.Tensor], batches: List[Tuple[int, int, int]],
                      uniform_lhs: Optional[torch.Tensor] = None, uniform_rhs: Optional[torch.Tensor] = None,
                      want_per_batch: bool = True, weights: Optional[torch.Tensor] = None) -> List[Stats]:
        """Trains the listed (offset, count, relation) batches of the edge arrays.  Edge arrays on
        the CPU are copied by the library (pin them to make the copy asynchronous).  `weights`:
        per-edge weights parallel to the edge arrays (EdgeList.weight), moved to the device here."""
        if not batches:
            return []
        if model.num_dynamic_rels == 0 and len(batches) > 1:
            relation_idx = batches[0][2]
            op_name = model.operator_of(relation_idx)
            wl, wr = model.tables_for(relation_idx)
            for r in {b[2] for b in batches}:
                if model.tables_for(r)[0] is not wl or model.tables_for(r)[1] is not wr or model.operator_of(r) != op_name:
                    raise NotImplementedError("batches of one call must read the same pair of tables through the same operator "
                                              "(process_in_batches cuts a list into such runs)")
        stats = self._train_run(model, lhs, rhs, rel, np.array(batches, dtype=_BATCH), uniform_lhs, uniform_rhs, want_per_batch, weights)
        if stats is None:
            return []
        return [Stats(loss=l, reg=g, violators_lhs=vl, violators_rhs=vr, count=n) for l, g, vl, vr, n in stats.tolist()]

    def _train_run(self, model: MultiRelationEmbedder, lhs, rhs, rel, batches: np.ndarray, uniform_lhs=None, uniform_rhs=None,
                   want_stats: bool = True, weights: Optional[torch.Tensor] = None) -> Optional[np.ndarray]:
        """One library call over _BATCH records that read one pair of tables through one operator; the _STATS records of
        the batches, or None when they are not wanted."""
        dyn = model.num_dynamic_rels > 0
        rels = [0] if dyn else np.unique(batches["rel"]).tolist()
        nat, bucket, local = self._bound(model, 0 if dyn else int(batches["rel"][0]), rels, int(batches["count"].max()))
        if local is not None:
            batches = batches.copy()
            batches["rel"] = local[batches["rel"]] if not dyn else 0
        stats = np.empty(len(batches), dtype=_STATS) if want_stats else None
        self._call(nat, bucket, model, lhs, rhs, rel, batches.ctypes.data, len(batches), uniform_lhs, uniform_rhs,
                   stats.ctypes.data if want_stats else None, weights)
        return stats

    def _bound(self, model, relation_idx: int, rels, max_count: int):
        """(context, bucket structure, place of every relation in its operator group -- or None where it is its index) for
        batches of relations `rels`, which read the tables of `relation_idx`."""
        for r in rels:
            if model.relations[r].all_negs:
                raise NotImplementedError("relations with all_negs=True are not trained by torchbiggraph_b200 (the evaluator ranks them)")
        op_name = model.operator_of(relation_idx)
        nat = self._context(model, max_count, op_name)
        wl, wr = model.tables_for(relation_idx)
        al, ar = self._op_states(model, op_name)
        gl = self._state_for(wl)
        states = (gl, gl if wr is wl else self._state_for(wr), al, ar)
        gl_, gr_ = model.globals_for(relation_idx)
        if gl_ is not None:
            if not isinstance(self.model_optimizer, AsyncAdagrad):
                raise RuntimeError("the model has global embeddings but model_optimizer is not an AsyncAdagrad over them")
            states = states + (self.model_optimizer.sum_for(gl_), self.model_optimizer.sum_for(gr_))
        # the library indexes operator rows and relation weights by the relation's place in its operator group
        dyn = model.num_dynamic_rels > 0
        members = [0] if dyn else model.op_groups[op_name]
        bucket = nat.bucket(model, relation_idx, states, [self.relation_weights[g] for g in members])
        if dyn or len(members) != len(model.relations):
            return nat, bucket, np.array([g[1] for g in model.group_of], dtype=np.int32)
        return nat, bucket, None

    def _call(self, nat, bucket, model, lhs, rhs, rel, batches: int, num_batches: int, uniform_lhs, uniform_rhs, stats: Optional[int], weights):
        """pbg_train_batches, or with edges on the host pbg_train_batches_host; `batches` and `stats` are addresses."""
        on_host = lhs.device.type == "cpu"
        fn = nat.lib.pbg_train_batches_host if on_host else nat.lib.pbg_train_batches
        for t in (lhs, rhs, rel, uniform_lhs, uniform_rhs):
            if t is not None and (t.dtype != torch.long or not t.is_contiguous() or (t.device.type == "cpu") != on_host):
                raise TypeError("edge and uniform-id arrays must be contiguous int64, all on the host or all on the device")
        self._calls += 1
        if weights is not None:
            if weights.shape[0] != lhs.shape[0]:
                raise ValueError("one weight per edge is needed")
            weights = weights.to(device=model.device, dtype=torch.float32).contiguous()     # kept alive until the call returns
            check(nat.lib.pbg_set_edge_weights(nat.ctx, _ptr(weights)), nat.ctx)
        check(nat.ordered(fn, C.byref(bucket), _ptr(lhs), _ptr(rhs), _ptr(rel), lhs.shape[0], batches, num_batches,
                          _ptr(uniform_lhs), _ptr(uniform_rhs), self.seed + self._calls, stats), nat.ctx)

    def read_stats(self) -> Stats:
        s = PbgBatchStats()
        check(self._native.lib.pbg_read_stats(self._native.ctx, C.byref(s)), self._native.ctx)
        return Stats(loss=float(s.loss), reg=float(s.reg), violators_lhs=int(s.violators_lhs),
                     violators_rhs=int(s.violators_rhs), count=int(s.count))

    # ---- the reference interface ---------------------------------------------------------------
    def _process_one_batch(self, model: MultiRelationEmbedder, batch_edges: EdgeList,
                           uniform_lhs=None, uniform_rhs=None) -> Stats:
        dyn = model.num_dynamic_rels > 0
        if dyn and batch_edges.has_scalar_relation_type():
            raise TypeError("Need relation for each positive pair")
        if not dyn and not batch_edges.has_scalar_relation_type():
            raise TypeError("All positive pairs must come from the same relation")
        n = len(batch_edges)
        if n == 0:
            return Stats(loss=0.0, reg=0.0, violators_lhs=0, violators_rhs=0, count=0)
        dev = model.device
        lhs = batch_edges.lhs.to_tensor().to(dev).contiguous()
        rhs = batch_edges.rhs.to_tensor().to(dev).contiguous()
        rel = batch_edges.rel.to(dev).contiguous() if dyn else None
        r = 0 if dyn else batch_edges.get_relation_type_as_scalar()
        nat, bucket, local = self._bound(model, r, (r,), n)
        ul = None if uniform_lhs is None else nat._uniform(uniform_lhs, dev)
        ur = None if uniform_rhs is None else nat._uniform(uniform_rhs, dev)
        wgt = torch.as_tensor(batch_edges.weight) if batch_edges.has_weight() else None
        b, s = PbgBatch(0, n, r if local is None else int(local[r])), PbgBatchStats()
        self._call(nat, bucket, model, lhs, rhs, rel, C.addressof(b), 1, ul, ur, C.addressof(s), wgt)
        return Stats(loss=s.loss, reg=s.reg, violators_lhs=s.violators_lhs, violators_rhs=s.violators_rhs, count=s.count)

    def process_one_batch(self, model, batch_edges, uniform_lhs=None, uniform_rhs=None) -> Stats:
        if self.overrides is not None:
            raise NotImplementedError("model overrides are not supported by torchbiggraph_b200")
        return self._process_one_batch(model, batch_edges, uniform_lhs, uniform_rhs)


class B200RankingEvaluator(AbstractBatchProcessor):
    """RankingEvaluator (torchbiggraph/eval.py:43-81) on the device: per batch the forward pass, the
    rank of every positive among its negatives on both sides, and Stats(loss, pos_rank, mrr, r1,
    r10, r50, auc, count) as sums the caller averages with Stats.average().  `overrides` takes the
    two keys the reference's evaluator overrides on the model (eval.py:165-172): num_batch_negs and
    num_uniform_negs."""

    def __init__(self, loss_fn: AbstractLossFunction, relation_weights: List[float], overrides=None):
        super().__init__(loss_fn, relation_weights, None)
        if getattr(loss_fn, "native_code", None) is None:
            raise NotImplementedError(f"loss function {type(loss_fn).__name__} has no device code (no CPU fallback)")
        unknown = set(overrides or {}) - {"num_batch_negs", "num_uniform_negs"}
        if unknown:
            raise NotImplementedError(f"model overrides {sorted(unknown)} are not supported by torchbiggraph_b200")
        self.neg_overrides = dict(overrides or {})
        self._native: Optional[_Native] = None
        self._natives: Dict[str, _Native] = {}
        self._native_model = lambda: None
        self.seed = 0
        self._calls = 0

    def _context(self, model, need_batch, op_name=None):
        op_name = model.operator_name if op_name is None else op_name
        if self._native_model() is not model:
            self._natives = {}
            self._native_model = weakref.ref(model)
        nat = self._natives.get(op_name)
        if nat is None or nat.max_batch < need_batch:
            cfg = model.config
            nat = _Native(model, max(cfg.batch_size, need_batch), 1, cfg.precision, cfg.lr, cfg.relation_lr,
                          getattr(self.loss_fn, "margin", cfg.margin), loss_code=self.loss_fn.native_code,
                          num_batch_negs=self.neg_overrides.get("num_batch_negs"),
                          num_uniform_negs=self.neg_overrides.get("num_uniform_negs"), op_name=op_name)
            self._natives[op_name] = nat
        self._native = nat
        return nat

    def _process_one_batch(self, model: MultiRelationEmbedder, batch_edges: EdgeList, uniform_lhs=None, uniform_rhs=None) -> Stats:
        dyn = model.num_dynamic_rels > 0
        if dyn and batch_edges.has_scalar_relation_type():
            raise TypeError("Need relation for each positive pair")
        if not dyn and not batch_edges.has_scalar_relation_type():
            raise TypeError("All positive pairs must come from the same relation")
        n = len(batch_edges)
        if n == 0:
            return Stats(loss=0.0, pos_rank=0.0, mrr=0.0, r1=0.0, r10=0.0, r50=0.0, auc=0.0, count=0)
        dev = model.device
        r = 0 if dyn else batch_edges.get_relation_type_as_scalar()
        op_name = model.operator_of(r)
        nat = self._context(model, n, op_name)
        lhs = batch_edges.lhs.to_tensor().to(dev).contiguous()
        rhs = batch_edges.rhs.to_tensor().to(dev).contiguous()
        rel = batch_edges.rel.to(dev).contiguous() if dyn else None
        ul = None if uniform_lhs is None else nat._uniform(uniform_lhs, dev)
        ur = None if uniform_rhs is None else nat._uniform(uniform_rhs, dev)
        members = [0] if dyn else model.op_groups[op_name]
        bucket = nat.bucket(model, r, None, [self.relation_weights[g] for g in members])
        full_r, r = r, (0 if dyn else model.group_of[r][1])     # the library's relation index is local to the operator group
        out = _lib.PbgEvalStats()
        self._calls += 1
        if batch_edges.has_weight():                 # the evaluator's loss is weighted like the trainer's (eval.py:55-56)
            wgt = torch.as_tensor(batch_edges.weight).to(device=dev, dtype=torch.float32).contiguous()
            check(nat.lib.pbg_set_edge_weights(nat.ctx, _ptr(wgt)), nat.ctx)
        if model.relations[0 if dyn else full_r].all_negs:
            # every entity of a side's table is a negative (model.py:582-617): ranks among the whole partition
            st = nat.ordered(nat.lib.pbg_eval_batch_all_negs, C.byref(bucket), _ptr(lhs), _ptr(rhs), _ptr(rel), n, r,
                             self.seed + self._calls, C.byref(out))
            if st == _lib.PBG_ERR_UNSUPPORTED:
                raise NotImplementedError(nat.lib.pbg_last_error(nat.ctx).decode())
            check(st, nat.ctx)
        else:
            check(nat.ordered(nat.lib.pbg_eval_batch, C.byref(bucket), _ptr(lhs), _ptr(rhs), _ptr(rel), n, r, _ptr(ul), _ptr(ur),
                              self.seed + self._calls, C.byref(out)), nat.ctx)
        return Stats(loss=float(out.loss), pos_rank=out.pos_rank, mrr=out.mrr, r1=out.r1, r10=out.r10, r50=out.r50,
                     auc=out.auc, count=int(out.count))

    def process_one_batch(self, model, batch_edges, uniform_lhs=None, uniform_rhs=None) -> Stats:
        return self._process_one_batch(model, batch_edges, uniform_lhs, uniform_rhs)


def _draw_batches(counts: List[int], batch_size: int, generator=None) -> List[Tuple[int, int, int]]:
    """Batch descriptors over edges sorted by relation (counts[r] edges of relation r): repeatedly pick a relation with
    probability proportional to its remaining edges and emit its next <= batch_size edges (batching.py:58-79).
    The pick is an exponential race -- relation r arrives after Exp(1) / remaining[r], the first one wins (Efraimidis and
    Spirakis, weighted random sampling) -- which takes the same draws as torch.multinomial and gives the same picks at a
    fraction of its overhead; it runs once per batch."""
    rels = [r for r, n in enumerate(counts) if n > 0]
    remaining = [counts[r] for r in rels]
    starts = np.concatenate([[0], np.cumsum(remaining)[:-1]]).astype(np.int64).tolist()
    left = np.array(remaining, dtype=np.float32)
    arrival = torch.empty(len(rels), dtype=torch.float32)
    speed = arrival.numpy()
    out = []
    total = sum(remaining)
    while total > 0:
        arrival.exponential_(1, generator=generator)
        with np.errstate(divide="ignore"):
            np.divide(left, speed, out=speed)
        i = int(speed.argmax())
        n = min(batch_size, remaining[i])
        out.append((starts[i], n, rels[i]))
        starts[i] += n
        remaining[i] -= n
        left[i] = remaining[i]
        total -= n
    return out


def _batches_group_by_relation(rel_sorted: torch.Tensor, batch_size: int, generator=None):
    """The same over the sorted relation ids themselves."""
    return _draw_batches(torch.bincount(rel_sorted, minlength=1).tolist(), batch_size, generator)


def process_in_batches(batch_size: int, model: MultiRelationEmbedder, batch_processor: B200Trainer,
                       edges: EdgeList, indices: Optional[torch.Tensor] = None, delay: float = 0.0) -> Stats:
    """torchbiggraph/batching.py:91-125 with the batch loop moved onto the device.  Per-edge weights
    (EdgeList.weight) travel with the edges.  With standard relations the batches come in the
    reference's order (batching.py:58-79); consecutive batches that read the same pair of embedding
    tables go to the library in one call, so relations over different entity types simply cut the
    list into more calls."""
    if indices is not None:
        edges = edges[indices]
    if delay > 0:
        time.sleep(delay)
    n = len(edges)
    if n == 0:
        return Stats(count=0)
    lhs, rhs = edges.lhs.to_tensor().contiguous(), edges.rhs.to_tensor().contiguous()
    weights = torch.as_tensor(edges.weight) if edges.has_weight() else None
    rel = None
    if model.num_dynamic_rels > 0:
        rel = edges.get_relation_type_as_vector().contiguous()
        batches = _even_batches(n, batch_size, 0)
    elif edges.has_scalar_relation_type():
        batches = _even_batches(n, batch_size, edges.get_relation_type_as_scalar())
    else:
        # sorted by relation on the device, wherever the edges are: it is a fraction of the copy there
        dev = model.device
        counts = torch.bincount(edges.rel, minlength=1).tolist()
        order = torch.argsort(edges.rel.to(dev, non_blocking=True), stable=True)
        lhs, rhs = lhs.to(dev, non_blocking=True)[order], rhs.to(dev, non_blocking=True)[order]
        if weights is not None:
            weights = weights.to(dev, non_blocking=True)[order]
        batches = np.array(_draw_batches(counts, batch_size), dtype=_BATCH)
    runs = _runs_by_table_pair(model, batches)
    stats = [batch_processor._train_run(model, lhs, rhs, rel, run, weights=weights) for run in runs]
    s = stats[0] if len(stats) == 1 else np.concatenate(stats)
    return Stats(loss=float(s["loss"].sum(dtype=np.float64)), reg=float(s["reg"].sum(dtype=np.float64)),
                 violators_lhs=int(s["violators_lhs"].sum()), violators_rhs=int(s["violators_rhs"].sum()), count=int(s["count"].sum()))


def _runs_by_table_pair(model: MultiRelationEmbedder, batches):
    """Cuts a batch list (tuples or _BATCH records) into maximal runs of consecutive batches whose relations read the same
    (lhs table, rhs table) pair through the same operator; one library call trains one run."""
    if model.num_dynamic_rels > 0 or len(batches) < 2:
        return [batches] if len(batches) else []
    rels = batches["rel"] if isinstance(batches, np.ndarray) else np.array([b[2] for b in batches])
    pairs: Dict[Tuple, int] = {}
    group = np.zeros(int(rels.max()) + 1, dtype=np.int64)
    for r in np.unique(rels).tolist():
        wl, wr = model.tables_for(r)
        group[r] = pairs.setdefault((wl.data_ptr(), wr.data_ptr(), model.operator_of(r)), len(pairs))
    cuts = [0] + (np.flatnonzero(np.diff(group[rels])) + 1).tolist() + [len(batches)]
    return [batches[a:b] for a, b in zip(cuts, cuts[1:])]
