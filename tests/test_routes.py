"""Which kernels a context takes for its training and its scores, by size and tier.  On the CPU (fake_cuda_util)."""
import os
import sys

import pytest

import fake_cuda_util as F


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    return F.build_fake(tmp_path_factory.mktemp("fake"))


# precision, comparator, dynamic, dimension, batch + uniform negatives, blocks of a wave; one kernel for training, for scores
ROUTES = [
    ("fp32", "cos", False, 256, 64, 64, 28, True, True),
    ("fp32", "cos", False, 256, 64, 65, 28, False, False),               # a fifth tile
    ("fp32", "cos", False, 260, 64, 64, 28, False, False),
    ("fp32", "dot", False, 100, 50, 50, 29, False, False),
    ("tf32x3", "dot", False, 128, 64, 64, 28, True, True),
    ("tf32x3", "dot", False, 132, 64, 64, 28, False, False),
    ("tf32x3", "dot", True, 104, 32, 0, 28, True, True),
    ("tf32x3", "dot", True, 104, 32, 1, 28, False, False),
    ("bf16x3", "cos", False, 100, 10, 5, 10, False, False),
    ("bf16x3", "l2", False, 100, 64, 64, 10, True, True),
    # a single pass of TF32 products: training's separate kernels are shorter from 33 columns on, from 13 blocks
    ("tf32", "dot", False, 100, 16, 16, 28, True, True),
    ("tf32", "cos", False, 100, 16, 17, 13, False, True),
    ("tf32", "cos", False, 100, 32, 32, 12, True, True),
    ("tf32", "dot", False, 100, 32, 33, 2, False, True),
    ("tf32", "dot", False, 100, 64, 64, 20, False, True),
    ("tf32", "l2", False, 100, 64, 64, 28, True, True),
    ("tf32", "dot", True, 104, 32, 0, 28, True, True),
]


def test_small_waves_take_one_kernel_where_it_is_shorter(fake):
    F.run_child(__file__, fake)


@pytest.mark.parametrize("clusters", [True, False])
def test_sorts_go_without_clusters_where_the_device_has_no_room_for_them(fake, clusters):
    """(with part of a device's SMs there may be none): the radix passes, not a launch that fails."""
    F.run_child(__file__, fake, "clusters" if clusters else "none", **({} if clusters else {"FAKE_NO_CLUSTERS": "1"}))


@pytest.mark.parametrize("kernel", ["chunk_kernel", "sort_waves_kernel"])
def test_a_kernel_the_device_cannot_hold_fails_no_call(fake, kernel):
    """(its opt-in to shared memory is refused when the context asks): the other kernels, and no error left for the next call."""
    F.run_child(__file__, fake, "without", FAKE_REFUSED=kernel)


def without(fake_so):
    import numpy as np
    fake, L, lib = F.load(fake_so)
    n, D = 300, 32
    ctx, bk, ids = F.create(L, lib, dim=D, op=0, comparator=0, loss=2, num_batch_negs=20, num_uniform_negs=10, max_batch_size=n), F.bucket(L, 400, D, False), F.dev(n, np.int64)
    for _ in range(2):
        fake.fake_arm(0, 0)
        assert F.train(L, lib, ctx, bk, ids, n, 1) == L.PBG_OK, lib.pbg_last_error(ctx)
        names = fake.fake_launched().decode()
        assert os.environ["FAKE_REFUSED"] not in names and "narrow_tile_kernel" in names, names


def sorts(fake_so, room):
    import numpy as np
    fake, L, lib = F.load(fake_so)
    n, rows, D = 300, 400, 32
    ids, W, G, p = F.dev(n, np.int64), F.dev((rows, D), np.float32), F.dev(rows, np.float32), F.p
    ctx = F.create(L, lib, dim=D, op=0, comparator=0, loss=2, num_batch_negs=20, num_uniform_negs=10, max_batch_size=n)
    bk = F.bucket(L, rows, D, False)
    for call in (lambda: F.train(L, lib, ctx, bk, ids, n, 1), lambda: lib.pbg_row_adagrad(ctx, p(W), p(G), rows, p(ids), p(W), n, 0.1),
                 lambda: lib.pbg_row_adagrad_static(p(W), p(G), rows, D, p(ids), p(W), n, 0.1, None)):
        fake.fake_arm(0, 0)
        assert call() == L.PBG_OK
        names = fake.fake_launched().decode()
        assert ("sort_waves_kernel" in names or "sort_rows_kernel" in names) == (room == "clusters"), names
        assert ("radix_scatter" in names) == (room != "clusters"), names


def main(fake_so, room=None):
    if room:
        return without(fake_so) if room == "without" else sorts(fake_so, room)
    import numpy as np
    fake, L, lib = F.load(fake_so)
    for precision, comp, dynamic, D, nb, nu, blocks, train, score in ROUTES:
        n = nb * blocks
        ctx = F.create(L, lib, dim=D, op=1, comparator=L.COMPARATOR_CODES[comp], loss=2, dynamic_relations=int(dynamic), num_batch_negs=nb,
                       num_uniform_negs=nu, precision=L.PRECISION_CODES[precision], max_batch_size=n)
        bk, ids = F.bucket(L, 400, D, dynamic), F.dev(n, np.int64)
        got = []
        for call in (lambda: F.train(L, lib, ctx, bk, ids, n, 1), lambda: F.score(lib, ctx, bk, ids, nb + nu)):
            fake.fake_arm(0, 0)
            assert call() == L.PBG_OK
            names = fake.fake_launched().decode()
            assert ("chunk_kernel" in names) != ("13gather_" in names), names
            got.append("chunk_kernel" in names)
        assert got == [train, score], (precision, comp, dynamic, D, nb, nu, blocks, got)


if __name__ == "__main__":
    main(*sys.argv[1:])
