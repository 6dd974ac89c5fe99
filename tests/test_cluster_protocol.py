"""Kernels that access the shared memory of the other CTAs of their cluster: a CTA's shared
memory exists for its peers only once it has started, so every such kernel passes a cluster
barrier before its first access to a peer.  Read from the sources, as a lost store or a fault
depends on when CTAs start."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "acousticscattering.jl_gb300", "csrc")
ACCESS = re.compile(r"\b(?:st_peer|ld_peer)_?\w*\s*(?:<\w+>)?\(")
BARRIER = re.compile(r"\bcluster_(?:sync_all|wait)\(\)")


def _kernels():
    """(file, kernel name, body) of every kernel that accesses a peer's shared memory."""
    out = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, end = 0, start
            for end in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            body = text[start:end]
            if ACCESS.search(body):
                out.append((name, m.group(1), body))
    return out


def test_kernels_are_found():
    assert any(k == "k_getf2_reg" for _, k, _ in _kernels())


@pytest.mark.parametrize("name,kernel,body", _kernels(), ids=lambda v: v if len(v) < 40 else "")
def test_barrier_before_the_first_access(name, kernel, body):
    first = ACCESS.search(body).start()
    assert BARRIER.search(body[:first]), f"{kernel}: peer access before any cluster barrier"
    assert body.count("cluster_arrive()") == body.count("cluster_wait()")
