"""A kernel that writes into other CTAs' shared memory first waits until every
CTA of its cluster runs: a cluster barrier, arrived at by all, before the first
remote store. (Read from the source: a start that is missed shows in no
result, until a CTA starts late.)"""

import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "galactic-tides_gb300" / "csrc"


def kernels(text):
    """(name, body) of every __global__ function, comments left out."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        start = text.index("{", m.end())
        depth, end = 1, start + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), text[start:end]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_remote_shared_memory_after_the_cluster_has_started(path):
    for name, body in kernels(path.read_text()):
        if "remote(" not in body:
            continue
        before = body[:body.index("remote(")]
        synced = "cluster_sync()" in before
        split = re.search(r"cluster_arrive\(\).*cluster_wait\(\)", before, re.S)
        assert synced or split, name


def test_the_cluster_sort_is_seen():
    names = [n for n, body in kernels((CSRC / "radix_sort.cu").read_text()) if "remote(" in body]
    assert names == ["k_sort_cluster"]
