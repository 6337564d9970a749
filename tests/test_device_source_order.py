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


def test_a_launch_that_does_not_wait_acquires_what_the_one_before_released():
    """Programmatic launches: griddepcontrol.wait makes the results of earlier launches visible to the grid that executes it.
    A kernel that starts without it (a sibling) has to take them over from the launch that did wait: release there, acquire
    here, and no reads through the read-only path, which that order does not cover."""
    common = _source("pbg_common.cuh")
    opens = _body(common, r"\bpdl_begin_open\([^;{]*\{")
    assert opens.index("pdl_wait()") < opens.index("st.release.gpu") < opens.index("pdl_release()")
    enter = _body(common, r"\bseam_enter\([^;{]*\{")
    assert enter.index("ld.acquire.gpu") < enter.index("pdl_wait()") < enter.index("fence.proxy.async.global")
    # pdl_release() alone (outside of the begin functions): only in front of seam_enter
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        source = _source(os.path.basename(path))
        for m in re.finditer(r"pdl_release\(\)", source):
            assert "seam_enter(" in source[m.end():m.end() + 300], (os.path.basename(path), source[m.start() - 200:m.end()])
    update = _source("pbg_update.cu")
    for kernel in ("tile_update_kernel", "hub_kernel"):              # the operator rows' instantiations are siblings
        body = _body(update, r"\b%s\(WaveDims[^;{]*\{" % kernel)
        assert not re.search(r"\b(keys|vals|hubcnt|hublist|biglist)\[(?!atomicAdd)", body), kernel
