"""Calls of the library over a CUDA runtime without a device (fake_cudart.cpp, fake_launch.cu), in a process of their own."""
import ctypes as C
import importlib.util
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "pytorch-biggraph_b200")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def build_fake(directory):
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    so = os.path.join(str(directory), "libfake_cudart.so")
    subprocess.check_call([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-cudart", "none", "-Xcompiler", "-fPIC", "-Xlinker",
                           "-soname=libcudart.so.12", "-I", os.path.join(PKG, "csrc"), os.path.join(HERE, "fake_cudart.cpp"),
                           os.path.join(HERE, "fake_launch.cu"), "-o", so])
    return so


def run_child(script, fake_so, *args, **env):
    out = subprocess.run([sys.executable, os.path.abspath(script), fake_so, *args], env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout[-3000:] + out.stderr[-3000:]


def load(fake_so):
    """In the child: the fake runtime, the binding's module, the library on top of the fake."""
    fake = C.CDLL(fake_so, mode=C.RTLD_GLOBAL)
    fake.fake_launched.restype = C.c_char_p
    spec = importlib.util.spec_from_file_location("pbg_lib", os.path.join(PKG, "torchbiggraph_b200", "_lib.py"))
    L = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(L)
    return fake, L, L.lib()


def create(L, lib, **kw):
    cfg = L.PbgConfig(**dict(dict(num_rels=5, batches_in_flight=1, margin=0.1, lr=0.1, relation_lr=0.1), **kw))
    ctx = C.c_void_p()
    assert lib.pbg_create(C.byref(cfg), 0, None, C.byref(ctx)) == 0, lib.pbg_last_error(ctx)
    return ctx


_keep = []


def dev(shape, dtype):
    """Zeros in "device" memory, aligned as cudaMalloc's, for as long as the process lives."""
    import numpy as np
    size = int(np.prod(shape)) * np.dtype(dtype).itemsize
    raw = np.zeros(size + 256, np.uint8)
    _keep.append(raw)
    return raw[-raw.ctypes.data % 256:][:size].view(dtype).reshape(shape)


def p(a):
    return a.ctypes.data_as(C.c_void_p)


def bucket(L, rows, D, dynamic):
    import numpy as np
    W, G, op, ops = dev((rows, D), np.float32), dev(rows, np.float32), dev((5, D), np.float32), dev((5, D), np.float32)
    return L.PbgBucket(lhs_emb=W.ctypes.data, lhs_state=G.ctypes.data, lhs_rows=rows, rhs_emb=W.ctypes.data, rhs_state=G.ctypes.data, rhs_rows=rows,
                       rhs_op=op.ctypes.data, rhs_op_state=ops.ctypes.data, lhs_op=op.ctypes.data if dynamic else None, lhs_op_state=ops.ctypes.data if dynamic else None)


def train(L, lib, ctx, bk, ids, batch, nbatches):
    batches, stats = (L.PbgBatch * nbatches)(*[L.PbgBatch(batch * i, batch, 0) for i in range(nbatches)]), (L.PbgBatchStats * nbatches)()
    return lib.pbg_train_batches(ctx, C.byref(bk), p(ids), p(ids), p(ids), len(ids), C.addressof(batches), nbatches, None, None, 7, C.addressof(stats))


def score(lib, ctx, bk, ids, cols):
    import numpy as np
    pos, neg = dev(len(ids), np.float32), dev((len(ids), cols), np.float32)
    return lib.pbg_score_batch(ctx, C.byref(bk), p(ids), p(ids), p(ids), len(ids), 0, None, None, 7, p(pos), p(pos), p(neg), p(neg))
