"""Kernels that store into other blocks' shared memory: a barrier of the cluster comes before the first remote
access (a block that has not started has no shared memory to write to).  Read from the sources, on the CPU."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "simple-dftd3_b200" / "csrc"


def _kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
            start = text.index("{", m.end())
            depth, at = 1, start + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            body = text[start:at]
            if "this_cluster" in body:
                yield pytest.param(body, id=f"{path.stem}-{m.group(1)}")


@pytest.mark.parametrize("body", list(_kernels()))
def test_barrier_before_first_remote_access(body):
    # mol_reduce writes to rank 0's shared memory
    remote = [m.start() for m in re.finditer(r"map_shared_rank|mol_reduce<", body)]
    barriers = [m.start() for m in re.finditer(r"cluster\.sync\(\)|mol_cluster_wait\(\)", body)]
    assert remote and barriers
    assert barriers[0] < remote[0]
    if "mol_cluster_wait" in body:
        assert body.index("mol_cluster_arrive()") < body.index("mol_cluster_wait()")


def test_finds_the_kernels():
    assert len(list(_kernels())) >= 2
