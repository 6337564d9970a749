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


@pytest.fixture(scope="module")
def context():
    from torchbiggraph_b200 import _lib
    L = _lib.lib()
    cfg = _lib.PbgConfig(dim=4, op=0, comparator=0, loss=2, dynamic_relations=0, num_rels=1, num_batch_negs=50, num_uniform_negs=50,
                         precision=0, max_batch_size=5000, batches_in_flight=14, lr=0.1, relation_lr=0.1)   # lists of up to 280,000
    ctx = C.c_void_p()
    assert L.pbg_create(C.byref(cfg), torch.cuda.current_device(), None, C.byref(ctx)) == 0
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
