"""Kernels of thread-block clusters that write to their peers' shared memory: the programming model
leaves such an access undefined until every CTA of the cluster has started, so each of them
has to pass a whole cluster barrier before the first one.  A missing barrier is a race that no
run shows reliably, so the order is read from the source: the wait stands ahead of the loop with
the kernel's remote accesses, outside every block."""
import os
import re

import pytest

from conftest import PKG_ROOT


def _body(file, kernel):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(PKG_ROOT, "csrc", file)).read())
    start = text.index("{", text.index("\n" + kernel + "("))
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start + 1:i]
    raise AssertionError(kernel)


@pytest.mark.parametrize("file,kernel,loop,remote", [
    ("heev.cu", "k_hetrd_panel_c", "for (int j = -1;", "panel_peer("),
    ("tridiag_dc.cuh", "k_dc_merge", "for (int s = coop", "share("),
])
def test_cluster_barrier_before_remote_access(file, kernel, loop, remote):
    body = _body(file, kernel)
    ahead = body[:body.index(loop)]
    assert remote in body and remote not in ahead
    arrive, wait = ahead.find("cluster_arrive();"), ahead.rfind("cluster_wait();")
    assert 0 <= arrive < wait, "no cluster barrier before the loop with the remote accesses"
    for at in (arrive, wait):   # every CTA of a cluster passes it
        assert ahead[:at].count("{") == ahead[:at].count("}")
