"""The one-kernel cluster sort behind the optimizer steps, at the edges of its shapes: one CTA, the last list of a cluster
size and the first of the next, 4 / 8 / 16 pairs per thread, and the list too long for it.  Driven through
pbg_row_adagrad (duplicates must meet, whatever their distance), against a plain PyTorch step."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _create(**options):
    from torchbiggraph_b200 import _lib
    L = _lib.lib()
    cfg = _lib.PbgConfig(dim=4, op=0, comparator=0, loss=2, dynamic_relations=0, num_rels=1, num_batch_negs=50, num_uniform_negs=50,
                         precision=0, max_batch_size=5000, batches_in_flight=14, lr=0.1, relation_lr=0.1)   # lists of up to 280,000
    for name, value in options.items():
        setattr(cfg, name, value)
    ctx = C.c_void_p()
    assert L.pbg_create(C.byref(cfg), torch.cuda.current_device(), None, C.byref(ctx)) == 0
    return L, ctx


@pytest.fixture(scope="module")
def context():
    L, ctx = _create()
    yield L, ctx
    L.pbg_destroy(ctx)


@pytest.mark.parametrize("n", [1, 33, 4096, 4097, 16384, 16385, 65536, 65537, 131073, 262144, 262145])
@pytest.mark.parametrize("rows", [200, 100_000, 3_000_000])
def test_duplicates_meet_at_every_list_shape(context, n, rows):
    L, ctx = context
    rng = np.random.default_rng(n + rows)
    ids = torch.tensor(rng.integers(0, rows, n)).cuda()
    grads = torch.tensor(rng.integers(-3, 4, (n, 4)).astype(np.float32)).cuda()          # integers: sums are exact in any order
    W, G = torch.zeros(rows, 4, device="cuda"), torch.full((rows,), 0.25, device="cuda")
    assert L.pbg_row_adagrad(ctx, _ptr(W), _ptr(G), rows, _ptr(ids), _ptr(grads), n, 0.1) == 0
    total = torch.zeros(rows, 4, device="cuda").index_add_(0, ids, grads)
    want_G = 0.25 + (total * total).mean(1)
    torch.testing.assert_close(G, want_G, rtol=1e-6, atol=0)
    torch.testing.assert_close(W, -0.1 * total / (want_G.sqrt() + 1e-10)[:, None], rtol=1e-5, atol=1e-7)


def test_ids_outside_the_table_are_reported_and_skipped(context):
    from torchbiggraph_b200 import _lib
    L, ctx = context
    n, rows = 5000, 1000
    ids = torch.arange(n, device="cuda") % rows
    ids[17], ids[4999] = rows, -1
    grads = torch.ones(n, 4, device="cuda")
    W, G = torch.zeros(rows, 4, device="cuda"), torch.zeros(rows, device="cuda")
    assert L.pbg_row_adagrad(ctx, _ptr(W), _ptr(G), rows, _ptr(ids), _ptr(grads), n, 0.1) == _lib.PBG_ERR_INDEX_RANGE
    want = torch.full((rows,), 25.0, device="cuda")                                       # five gradients of ones: mean square 25
    want[17], want[999] = 16.0, 16.0
    torch.testing.assert_close(G, want)


def _train(rows_told=None, batches=30):
    """(table, state, launches) after `batches` batches of 1000 edges on 3000 rows at four in flight: eight waves.  No uniform
    negatives, so no row but the edges' own is touched, however many rows the library is told of."""
    from torchbiggraph_b200 import _lib
    L, ctx = _create(max_batch_size=1000, batches_in_flight=4, num_uniform_negs=0)
    rows = 3000
    g = torch.Generator().manual_seed(3)
    W, G = torch.randn(rows, 4, generator=g).cuda(), torch.rand(rows, generator=g).cuda()
    lhs, rhs = ((torch.rand(1000 * batches, generator=g) ** 3 * rows).long().cuda() for _ in range(2))         # some rows a hub's size
    b = _lib.PbgBucket(lhs_emb=W.data_ptr(), lhs_state=G.data_ptr(), lhs_rows=rows_told or rows,
                       rhs_emb=W.data_ptr(), rhs_state=G.data_ptr(), rhs_rows=rows_told or rows)
    weights = (C.c_float * 1)(1.0)
    b.relation_weights = weights
    lists, stats = (_lib.PbgBatch * batches)(*[_lib.PbgBatch(i * 1000, 1000, 0) for i in range(batches)]), (_lib.PbgBatchStats * batches)()
    for _ in range(2):
        before = L.pbg_launch_count(ctx)
        assert L.pbg_train_batches(ctx, C.byref(b), _ptr(lhs), _ptr(rhs), None, 1000 * batches, C.byref(lists), batches, None, None, 7, C.byref(stats)) == 0
    launches = L.pbg_launch_count(ctx) - before
    L.pbg_destroy(ctx)
    return W.cpu(), G.cpu(), launches


def test_without_clusters_and_with_keys_beyond_32_bits_the_sort_takes_the_radix_passes(monkeypatch):
    """The same order, so the same bits.  PBG_CLUSTER_SORT=0 stands for a device that cannot hold the clusters (part of its SMs);
    2^33 rows need keys of 34 bits, for which a second scratch is made at the first call.  Keys of 12 bits take two passes of three
    launches, keys of 34 four, and the key build; the cluster kernel takes the eight waves in three launches."""
    W, G, launches = _train()
    monkeypatch.setenv("PBG_CLUSTER_SORT", "0")
    Wr, Gr, radix = _train()
    monkeypatch.delenv("PBG_CLUSTER_SORT")
    Wl, Gl, wide = _train(rows_told=2 ** 33)
    assert torch.equal(W, Wr) and torch.equal(G, Gr) and torch.equal(W, Wl) and torch.equal(G, Gl)
    assert radix - launches == 8 * 7 - 3 and wide - launches == 8 * 13 - 3


def test_sort_scratch_follows_what_the_waves_need():
    """Bytes per slot of the workspace, below and above the longest list a cluster sorts (262,144): below, eight lists of 12 bytes a
    slot and one scratch of 56 (pairs twice, counters); above, a second scratch, and no more lists: 96 - 56 bytes less."""
    def slope(small, large):
        size = {}
        for edges in (small, large):
            L, ctx = _create(max_batch_size=edges, batches_in_flight=1)
            size[edges] = L.pbg_workspace_bytes(ctx)
            L.pbg_destroy(ctx)
        return (size[large] - size[small]) / (4.0 * (large - small))          # 50 + 50 negatives a side: four slots an edge
    assert slope(25_000, 50_000) - slope(100_000, 200_000) == pytest.approx(40.0, abs=1.0)
