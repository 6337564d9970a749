"""Orders in the device sources that no run can show to be missing: what they prevent happens once in a million launches, if
the hardware lets it happen at all.  Checked on the text of csrc/ with its comments taken out, on the CPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pytorch-biggraph_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def _body(source, signature):
    """The function whose head `signature` matches up to its opening brace: from there to the brace that closes it."""
    at = source.index("{", re.search(signature, source).end() - 1)
    depth = 0
    for i in range(at, len(source)):
        depth += {"{": 1, "}": -1}.get(source[i], 0)
        if depth == 0:
            return source[at:i + 1]
    raise AssertionError("unbalanced braces")


def test_cluster_sort_waits_for_its_cluster_before_it_writes_to_another_cta():
    """CUDA: a CTA's shared memory may be accessed by its cluster once it has started -- a cluster barrier says so."""
    source = _source("pbg_sort.cu")
    body = _body(source, r"\bcluster_sort_body\([^;{]*\{")
    first_remote = body.index("map_shared_rank")
    waits = [m.start() for m in re.finditer(r"cluster\.(barrier_wait|sync)\(\)", body)]
    assert waits and waits[0] < first_remote
    users = [_body(source, r"\b%s\([^)]*\)\s*\{" % k) for k in ("sort_waves_kernel", "sort_rows_kernel")]
    assert source.count("cluster_sort_body<IPT>(") == len(users)
    for kernel in users:                                        # every thread arrives, whatever its part of the list
        assert kernel.index("barrier_arrive()") < min(kernel.index(w) for w in ("for (", "if (", "cluster_sort_body") if w in kernel)
