"""What a call leaves behind when one of its launches fails: an error, no launch behind the failed one, and every word and counter
that lives from call to call at zero, so that the next call is as good as the first.  On the CPU, under tests/fake_cudart.cpp."""
import ctypes as C
import importlib.util
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "pytorch-biggraph_b200")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.check_call([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "none", "-Xcompiler", "-fPIC", "-Xlinker",
                           "-soname=libcudart.so.12", "-I", os.path.join(PKG, "csrc"), os.path.join(HERE, "fake_cudart.cpp"),
                           os.path.join(HERE, "fake_launch.cu"), "-o", so])
    return so


CALLS = ["train", "train_small", "train_radix", "score", "eval", "eval_all", "row_adagrad", "randperm", "randperm_sorted", "sub_bucket", "sub_bucket_many"]


@pytest.mark.parametrize("call", CALLS)
def test_a_failed_launch_leaves_nothing_behind(fake, call):
    env = dict(os.environ)
    if call == "train_radix":
        env["PBG_CLUSTER_SORT"] = "0"
    out = subprocess.run([sys.executable, os.path.abspath(__file__), fake, call], env=env, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-3000:] + out.stderr[-3000:]


def _calls(L, lib, name):
    """A function that makes the call once and returns its status."""
    import numpy as np
    n, rows, D = 300, 400, 32
    dynamic = name.startswith("train") and name != "train_small"
    cfg = L.PbgConfig(dim=D, op=3 if dynamic else 2, comparator=0, loss=2, dynamic_relations=int(dynamic), num_rels=5, num_batch_negs=20, num_uniform_negs=10,
                      precision=L.PRECISION_CODES["fp32" if name == "train_small" else "tf32x3"], max_batch_size=100 if name.startswith("train") else n,
                      batches_in_flight=2 if dynamic else 1, margin=0.1, lr=0.1, relation_lr=0.1)
    ctx = C.c_void_p()
    assert lib.pbg_create(C.byref(cfg), 0, None, C.byref(ctx)) == 0, lib.pbg_last_error(ctx)
    keep = []

    def dev(shape, dtype):
        raw = np.zeros(int(np.prod(shape)) * np.dtype(dtype).itemsize + 256, np.uint8)
        a = raw[-raw.ctypes.data % 256:][:int(np.prod(shape)) * np.dtype(dtype).itemsize].view(dtype).reshape(shape)
        keep.append(a)
        return a

    def p(a):
        return a.ctypes.data_as(C.c_void_p)
    W, G, op, ops, ids = dev((rows, D), np.float32), dev(rows, np.float32), dev((5, D), np.float32), dev((5, D), np.float32), dev(n, np.int64)
    bk = L.PbgBucket(lhs_emb=W.ctypes.data, lhs_state=G.ctypes.data, lhs_rows=rows, rhs_emb=W.ctypes.data, rhs_state=G.ctypes.data, rhs_rows=rows,
                     rhs_op=op.ctypes.data, rhs_op_state=ops.ctypes.data, lhs_op=op.ctypes.data if dynamic else None, lhs_op_state=ops.ctypes.data if dynamic else None)
    ev = L.PbgEvalStats()
    if name.startswith("train"):
        batches, stats = (L.PbgBatch * 3)(*[L.PbgBatch(100 * i, 100, 0) for i in range(3)]), (L.PbgBatchStats * 3)()
        return lambda: lib.pbg_train_batches(ctx, C.byref(bk), p(ids), p(ids), p(ids), n, C.addressof(batches), 3, None, None, 7, C.addressof(stats))
    if name == "score":
        pos, neg = dev(n, np.float32), dev((n, 30), np.float32)
        return lambda: lib.pbg_score_batch(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, None, None, 7, p(pos), p(pos), p(neg), p(neg))
    if name == "eval":
        return lambda: lib.pbg_eval_batch(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, None, None, 7, C.byref(ev))
    if name == "eval_all":
        return lambda: lib.pbg_eval_batch_all_negs(ctx, C.byref(bk), p(ids), p(ids), None, n, 0, 7, C.byref(ev))
    if name == "row_adagrad":
        return lambda: lib.pbg_row_adagrad(ctx, p(W), p(G), rows, p(ids), p(W), n, 0.1)
    if name.startswith("randperm"):
        m = (1 << 22) + 1 if name == "randperm_sorted" else n
        out = dev(m, np.int64)
        return lambda: lib.pbg_randperm(ctx, m, 7, p(out))
    parts = 40 if name == "sub_bucket_many" else 2
    counts, perms, sizes = dev(parts * parts, np.int64), (C.c_void_p * 1)(dev(rows, np.int64).ctypes.data), (C.c_int64 * 1)(rows)
    return lambda: lib.pbg_sub_bucket(ctx, p(ids), p(ids), p(ids), n, 1, sizes, perms, sizes, perms, p(ids), p(ids), p(ids), parts, parts, 0,
                                      counts.ctypes.data_as(C.POINTER(C.c_int64)))


def main(fake_so, name):
    fake = C.CDLL(fake_so, mode=C.RTLD_GLOBAL)
    spec = importlib.util.spec_from_file_location("pbg_lib", os.path.join(PKG, "torchbiggraph_b200", "_lib.py"))
    L = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(L)
    lib = L.lib()
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
