"""The one-cluster pressure solver may write another block's shared memory only after a cluster
barrier that all its blocks have passed: before it, a block may not have started, and the write is
a device exception.  Blocks nearly always start together, so the order is checked in the source:
in the kernel's body an arrival and its wait stand before the first remote write.
"""
import os
import re

from polymps_gb300 import build


def _body(src, name):
    at = src.index("{", src.index(" " + name + "("))
    depth = 0
    for k in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[at:k + 1]


def test_cluster_barrier_before_the_first_remote_write():
    with open(os.path.join(build.CSRC, "mps_ppe.cu")) as f:
        body = re.sub(r"//[^\n]*", "", _body(f.read(), "k_cg_cluster"))
    # the lambda that publishes z writes where it is called
    body = re.sub(r"auto publish = .*?\n    };", "", body, flags=re.S)
    writes = [m.start() for m in re.finditer(r"\b(clPush<|publish\(|clStore\()", body)]
    assert writes
    arrive, wait = body.find("clArrive();"), body.find("clWait();")
    assert 0 <= arrive < wait < writes[0]
