"""What a call leaves behind when one of its launches fails: an error, no launch behind the failed one, and every word and counter
that lives from call to call at zero, so that the next call is as good as the first.  On the CPU (fake_cuda_util)."""
import ctypes as C
import sys

import pytest

import fake_cuda_util as F


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return F.build_fake(tmp_path_factory.mktemp("fake"))


CALLS = ["train", "train_small", "train_radix", "score", "eval", "eval_all", "row_adagrad", "randperm", "randperm_sorted", "sub_bucket", "sub_bucket_many"]


@pytest.mark.parametrize("call", CALLS)
def test_a_failed_launch_leaves_nothing_behind(fake, call):
    F.run_child(__file__, fake, call, **({"PBG_CLUSTER_SORT": "0"} if call == "train_radix" else {}))


def test_a_failed_allocation_is_the_failure_of_its_own_call(fake):
    """The runtime keeps an error until it is asked for it: the next call must not find it."""
    F.run_child(__file__, fake, "no_memory")


def test_scratch_that_could_not_grow_grows_at_the_next_call(fake):
    """Freed to make room for a larger one that the device had no memory for: the next call, of the old size, allocates it again."""
    F.run_child(__file__, fake, "no_growth")


def no_growth(fake, L, lib):
    import numpy as np
    n, rows, D = 4000, 400, 32
    ctx = F.create(L, lib, dim=D, op=2, comparator=0, loss=2, num_batch_negs=20, num_uniform_negs=10, precision=1, max_batch_size=100)
    ids, bk, p = F.dev(n, np.int64), F.bucket(L, rows, D, False), F.p

    def train_host(k):
        batches, stats = (L.PbgBatch * k)(*[L.PbgBatch(100 * i, 100, 0) for i in range(k)]), (L.PbgBatchStats * k)()
        neg = np.zeros((k, 5, 10), np.int64)
        return lib.pbg_train_batches_host(ctx, C.byref(bk), p(ids), p(ids), p(ids), 100 * k, C.addressof(batches), k, p(neg), p(neg), 7, C.addressof(stats))

    def split(relations):
        counts, perms, sizes = np.zeros(4, np.int64), (C.c_void_p * relations)(*[F.dev(rows, np.int64).ctypes.data] * relations), (C.c_int64 * relations)(*[rows] * relations)
        return lib.pbg_sub_bucket(ctx, p(ids), p(ids), p(ids), 300, relations, sizes, perms, sizes, perms, p(ids), p(ids), p(ids), 2, 2, 0,
                                  counts.ctypes.data_as(C.POINTER(C.c_int64)))
    for call, small, large in ((train_host, 2, 40), (split, 20, 300)):
        assert call(small) == L.PBG_OK
        fake.fake_no_memory(1)
        assert call(large) == L.PBG_ERR_CUDA
        fake.fake_no_memory(0)
        assert call(small) == L.PBG_OK and call(large) == L.PBG_OK


def no_memory(fake, L, lib):
    import numpy as np
    n, rows, D = 300, 400, 32
    ctx = F.create(L, lib, dim=D, op=2, comparator=0, loss=2, num_batch_negs=20, num_uniform_negs=10, precision=1, max_batch_size=n)
    ids, bk, p, ev = F.dev(n, np.int64), F.bucket(L, rows, D, False), F.p, L.PbgEvalStats()
    fake.fake_no_memory(1)                                       # (its scratch is allocated at its first call)
    assert lib.pbg_eval_batch_all_negs(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, 7, C.byref(ev)) == L.PBG_ERR_CUDA
    fake.fake_no_memory(0)
    assert F.train(L, lib, ctx, bk, ids, n, 1) == L.PBG_OK
    assert lib.pbg_eval_batch_all_negs(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, 7, C.byref(ev)) == L.PBG_OK


def _calls(L, lib, name):
    """A function that makes the call once and returns its status."""
    import numpy as np
    n, rows, D = 300, 400, 32
    dynamic = name.startswith("train") and name != "train_small"
    ctx = F.create(L, lib, dim=D, op=3 if dynamic else 2, comparator=0, loss=2, dynamic_relations=int(dynamic), num_batch_negs=20, num_uniform_negs=10,
                   precision=L.PRECISION_CODES["fp32" if name == "train_small" else "tf32x3"], max_batch_size=100 if name.startswith("train") else n,
                   batches_in_flight=2 if dynamic else 1)
    ids, bk, p, ev = F.dev(n, np.int64), F.bucket(L, rows, D, dynamic), F.p, L.PbgEvalStats()
    if name.startswith("train"):
        return lambda: F.train(L, lib, ctx, bk, ids, 100, 3)
    if name == "score":
        return lambda: F.score(lib, ctx, bk, ids, 30)
    if name == "eval":
        return lambda: lib.pbg_eval_batch(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, None, None, 7, C.byref(ev))
    if name == "eval_all":
        return lambda: lib.pbg_eval_batch_all_negs(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, 7, C.byref(ev))
    if name == "row_adagrad":
        W, G = F.dev((rows, D), np.float32), F.dev(rows, np.float32)
        return lambda: lib.pbg_row_adagrad(ctx, p(W), p(G), rows, p(ids), p(W), n, 0.1)
    if name.startswith("randperm"):
        m = (1 << 22) + 1 if name == "randperm_sorted" else n
        out = F.dev(m, np.int64)
        return lambda: lib.pbg_randperm(ctx, m, 7, p(out))
    parts = 40 if name == "sub_bucket_many" else 2
    counts, perms, sizes = F.dev(parts * parts, np.int64), (C.c_void_p * 1)(F.dev(rows, np.int64).ctypes.data), (C.c_int64 * 1)(rows)
    return lambda: lib.pbg_sub_bucket(ctx, p(ids), p(ids), p(ids), n, 1, sizes, perms, sizes, perms, p(ids), p(ids), p(ids), parts, parts, 0,
                                      counts.ctypes.data_as(C.POINTER(C.c_int64)))


def main(fake_so, name):
    fake, L, lib = F.load(fake_so)
    if name in ("no_memory", "no_growth"):
        return globals()[name](fake, L, lib)
    call = _calls(L, lib, name)
    fake.fake_arm(0, 0)
    assert call() == L.PBG_OK and fake.fake_unclean() == 0
    many = fake.fake_launches()
    assert many > 0
    for at in range(1, many + 1):
        fake.fake_arm(at, 1)
        assert call() == L.PBG_ERR_CUDA, at
        assert fake.fake_behind_failure() == 0, (at, fake.fake_behind_failure())
        for again in range(2):                                  # (counters are used in turn)
            fake.fake_arm(0, 0)
            rc = call()
            assert rc == L.PBG_OK and fake.fake_unclean() == 0 and fake.fake_launches() == many, (at, again, rc, fake.fake_unclean())


if __name__ == "__main__":
    main(*sys.argv[1:])
