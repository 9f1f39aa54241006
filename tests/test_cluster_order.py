"""Distributed shared memory may be touched only once every block of the cluster is known to run:
in each kernel that maps another block's shared memory, a wait at the cluster's barrier comes before
the first access through the mapped pointer, and another after the last.  Read from the source: the
order cannot be seen from results, which are right whenever the blocks happen to start in time."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fjmodels_gb300", "csrc")
WAIT = re.compile(r"\bcluster\.(?:sync|barrier_wait)\s*\(|barrier\.cluster\.wait")


def _kernels():
    """(file, name, body) of every kernel of the library, comments taken out"""
    for f in sorted(os.listdir(CSRC)):
        if not f.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, f)) as h:
            text = re.sub(r"//[^\n]*|/\*.*?\*/", "", h.read(), flags=re.S)
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield f, m.group(1), text[m.end():i]


MAPPED = [(f, n, b) for f, n, b in _kernels() if "map_shared_rank" in b]


def test_there_are_such_kernels():
    assert "k_poisson_cumulative" in [n for _, n, _ in MAPPED]


@pytest.mark.parametrize("name,body", [(n, b) for _, n, b in MAPPED], ids=[n for _, n, _ in MAPPED])
def test_waits_enclose_remote_accesses(name, body):
    for ptr in re.findall(r"(\w+)\s*=\s*cluster\.map_shared_rank", body):
        uses = [m.start() for m in re.finditer(rf"\b{ptr}\s*\[", body)]
        waits = [m.start() for m in WAIT.finditer(body)]
        assert uses and any(w < uses[0] for w in waits), f"{name}: {ptr} used before any block is known to run"
        assert any(w > uses[-1] for w in waits), f"{name}: {ptr} used after the last wait"
