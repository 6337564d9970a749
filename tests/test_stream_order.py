"""Calls made under another CUDA stream than the one a library context was created on: what PyTorch has queued on the caller's
stream (uploads, sorts, conversions of the arguments) comes first, and what it queues afterwards comes behind the call."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

import torchbiggraph_b200 as T
from torchbiggraph_b200 import trainer as trainer_module


class _Stream:
    def __init__(self, number, log):
        self.cuda_stream, self.log = number, log

    def wait_stream(self, other):
        self.log.append(f"{self.cuda_stream} waits for {other.cuda_stream}")


@pytest.mark.parametrize("current,want", [(1, ["call"]), (2, ["1 waits for 2", "call", "2 waits for 1"])], ids=["same", "other"])
@pytest.mark.parametrize("status", [0, 3], ids=["ok", "error"])
def test_library_calls_are_ordered_with_the_current_stream(monkeypatch, current, want, status):
    """(CPU: a library that only writes down when it is called)"""
    log = []

    def call(*args):
        log.append("call")
        return status
    nat = object.__new__(trainer_module._Native)
    nat.lib = SimpleNamespace(pbg_train_batches_host=call, pbg_destroy=lambda c: 0)
    nat.ctx, nat.device_index, nat.stream, nat.stream_handle = None, 0, _Stream(1, log), 1
    monkeypatch.setattr(trainer_module, "_current_stream", lambda device_index: current, raising=False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: _Stream(current, log))
    tr = T.B200Trainer(None, T.LOSS_FUNCTIONS.get_class("softmax")(margin=0.1), [1.0])
    e = torch.zeros(4, dtype=torch.long)
    try:
        tr._call(nat, trainer_module.PbgBucket(), None, e, e, None, 0, 1, None, None, None, None)
        assert status == 0
    except trainer_module._lib.PbgError:
        assert status != 0
    assert log == want


def _rig(seed=7, D=32, rows=500):
    rng = np.random.default_rng(seed)
    rels = [T.RelationSchema(f"r{i}", "e", "e", operator="translation") for i in range(3)]
    cfg = T.ConfigSchema(entities={"e": T.EntitySchema()}, relations=rels, dimension=D, comparator="dot", loss_fn="softmax", lr=0.1,
                         batch_size=100, num_batch_negs=50, num_uniform_negs=0)
    model = T.make_model(cfg, "cuda")
    W = torch.tensor((rng.standard_normal((rows, D)) * 0.1).astype(np.float32)).cuda()
    model.set_embeddings("e", T.Side.LHS, W)
    model.set_embeddings("e", T.Side.RHS, W)
    loss_fn = T.LOSS_FUNCTIONS.get_class("softmax")(margin=0.1)
    tr = T.B200Trainer(T.make_optimizer(cfg, model.parameters(), False), loss_fn, [1.0] * 3)
    tr.partitioned_optimizers["e", 0] = T.make_optimizer(cfg, [W], True)
    return model, tr, T.B200RankingEvaluator(loss_fn, [1.0] * 3), W


def _edges(n, rows, rel, pinned, weighted, seed=11):
    g = torch.Generator().manual_seed(seed)
    lhs, rhs = (torch.randint(0, rows, (n,), generator=g) for _ in range(2))
    rel = torch.randint(0, 3, (n,), generator=g) if rel is None else torch.tensor(rel)
    w = torch.rand(n, generator=g) + 0.5 if weighted else None
    if pinned:
        lhs, rhs, rel, w = (None if t is None else t.pin_memory() for t in (lhs, rhs, rel, w))
    return lhs, rhs, rel, w


def _calls(model, tr, ev, W, under):
    """Every kind of call once, each under `under()`; results and the tables they leave."""
    def edge_list(*a):
        lhs, rhs, rel, w = a
        return T.EdgeList(T.EntityList.from_tensor(lhs), T.EntityList.from_tensor(rhs), rel, w)
    out = []
    with under():                                            # several relations in host memory: sorted by PyTorch on the device
        torch.manual_seed(5)
        s = T.process_in_batches(100, model, tr, edge_list(*_edges(5000, W.shape[0], None, True, True)))
        out.append(torch.tensor([s.metrics["loss"], float(s.count)]))
    one = _edges(100, W.shape[0], 1, False, True, seed=13)
    lhs, rhs = (t.cuda().repeat_interleave(2) for t in one[:2])
    torch.cuda.synchronize()
    with under():                                            # device tensors that are not contiguous: copied by PyTorch
        s = tr.process_one_batch(model, edge_list(lhs[::2], rhs[::2], one[2], one[3].double().cuda()))
        out.append(torch.tensor([s.metrics["loss"], float(s.count)]))
    with under():
        s = ev.process_one_batch(model, edge_list(lhs[::2], rhs[::2], one[2], None))
        out.append(torch.tensor([s.metrics["loss"], s.metrics["pos_rank"]]))
    with under():
        out += [t.clone() for t in model.forward(edge_list(lhs[::2], rhs[::2], one[2], None))]
    with under():                                            # no statistics: the call returns before its kernels have run
        d = [t.cuda() for t in _edges(5000, W.shape[0], 0, False, True, seed=17)]
        tr.train_batches(model, d[0], d[1], None, [(i * 100, 100, 2) for i in range(50)], want_per_batch=False, weights=d[3].double())
        out += [W.clone(), tr.partitioned_optimizers["e", 0].sum_for(W).clone()]
        d = [t.fill_(0) for t in d]                          # (behind the call, which reads them)
    torch.cuda.synchronize()
    return [t.cpu() for t in out]


@pytest.mark.gpu
def test_calls_under_another_busy_stream_see_their_arguments():
    import contextlib
    want = _calls(*_rig(), under=contextlib.nullcontext)
    model, tr, ev, W = _rig()
    for f in (lambda: tr._context(model, 100), lambda: ev._context(model, 100)):
        f()                                                  # contexts on the default stream
    side = torch.cuda.Stream()

    @contextlib.contextmanager
    def busy():
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(40_000_000)                    # some 20 ms in front of whatever the call makes PyTorch queue
            yield
    got = _calls(model, tr, ev, W, under=busy)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"output {i}"


def test_shuffle_hands_over_a_permutation_that_is_complete_and_stays(monkeypatch):
    """A permutation that is not contiguous is copied by PyTorch: in front of the wait for PyTorch's stream, and kept until the
    library is done with it.  (CPU: a library that only writes down when it is called)"""
    import weakref

    from torchbiggraph_b200 import _C as native
    log, copies, contiguous = [], [], torch.Tensor.contiguous

    def copy(self, *a):
        out = contiguous(self, *a)
        log.append("copy")
        copies.append(weakref.ref(out))
        return out

    def call(*a):
        assert copies[-1]() is not None and a[-1] == copies[-1]().data_ptr()
        log.append("call")
        return 0
    monkeypatch.setattr(native, "_ctx", lambda device: None)
    monkeypatch.setattr(native, "_sync_torch", lambda device: log.append("wait"))
    monkeypatch.setattr(native._lib, "lib", lambda: SimpleNamespace(pbg_shuffle_rows=call))
    monkeypatch.setattr(torch.Tensor, "contiguous", copy)
    native.shuffle(torch.zeros(10, 3), torch.arange(20)[::2])
    assert log == ["copy", "wait", "call"]


def test_edge_list_utilities_use_a_context_for_one_thread_at_a_time(monkeypatch):
    """The reference's functions may run on several threads; here they share a device's context (one error word, scratch that
    grows).  (CPU: a library that writes down who is inside it)"""
    import threading
    import time

    from torchbiggraph_b200 import _C as native
    inside, most = [], []

    def call(*a):
        inside.append(1)
        most.append(len(inside))
        time.sleep(0.02)
        inside.pop()
        return 0
    fake = SimpleNamespace(pbg_shuffle_rows=call, pbg_reverse_permutation=call, pbg_randperm=call, pbg_sub_bucket=call)
    monkeypatch.setattr(native, "_ctx", lambda device: None)
    monkeypatch.setattr(native, "_sync_torch", lambda device: None)
    monkeypatch.setattr(native._lib, "lib", lambda: fake)
    e = torch.zeros(4, dtype=torch.long)
    calls = [lambda: native.randperm(4, seed=1, device="cpu"), lambda: native.reverse_permutation(e), lambda: native.shuffle(torch.zeros(4, 2), e),
             lambda: native.sub_bucket(e, e, e, [4], [e], [4], [e], e.clone(), e.clone(), e.clone(), 1, 1)]
    threads = [threading.Thread(target=c) for c in calls * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(most) == 8 and max(most) == 1
