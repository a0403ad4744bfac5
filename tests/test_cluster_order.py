"""Kernels on thread-block clusters, by their source: another CTA's shared memory is touched only behind a cluster barrier, since
nothing else says that the CTA has started.  (That order cannot be made to fail on a GPU at will.)"""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "tilert_b200" / "csrc"
REMOTE = r"\b(?:cluster_store|cluster_add|cluster_add_get|mbar_arrive_cluster|tma_load_2d_pair|umma_commit_pair)\s*\("


def cluster_kernels():
    """(name, body without comments) of every kernel launched as a cluster."""
    for path in sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__ void __cluster_dims__", text):
            name = re.search(r"(\w+_kernel)\(", text[m.start():]).group(1)
            start = end = text.index("{", m.start())
            level = 0
            while level > 0 or end == start:
                level += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield pytest.param(text[start: end], id=name)


@pytest.mark.parametrize("body", list(cluster_kernels()))
def test_a_barrier_comes_before_another_ctas_memory(body):
    remote = re.search(REMOTE, body)
    passed = re.search(r"\bcluster_(?:sync_all|wait)\(\)", body)
    assert remote and passed and passed.start() < remote.start()
    halves = [m.group(1) for m in re.finditer(r"\bcluster_(arrive|wait)\(\)", body)]
    assert halves in ([], ["arrive", "wait"])  # every thread that arrives waits, once


def test_the_kernels_are_found():
    assert {p.id for p in cluster_kernels()} >= {"greedy_kernel", "sample_kernel", "gemm_pair_kernel"}
