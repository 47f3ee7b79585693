"""Order of the accesses to another CTA's shared memory in the kernels' sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "ferrite_b200" / "csrc"
REMOTE = re.compile(r"\bst_cluster_\w+\(|\bld_cluster_\w+\(|\bmapa\b|cluster_map_shared_rank")


def kernels():
    for path in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]):
        src = re.sub(r"//[^\n]*", "", path.read_text())
        src = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", src)
        for m in re.finditer(r"__global__\s+void\s+(\w+)\s*\([^;{]*\)\s*\{", src):
            depth, end = 1, m.end()
            while depth and end < len(src):
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            yield path.name, m.group(1), src[m.end():end]


CASES = [(f, k, body) for f, k, body in kernels() if REMOTE.search(body)]


@pytest.mark.parametrize("file,kernel,body", CASES, ids=[f"{f}:{k}" for f, k, _ in CASES])
def test_a_cluster_has_started_before_its_shared_memory_is_touched(file, kernel, body):
    """Distributed shared memory may be accessed once all CTAs of the cluster run, which a barrier of the cluster that was met before shows."""
    before = body[:REMOTE.search(body).start()]
    assert "cluster_arrive();" in before and "cluster_wait();" in before[before.index("cluster_arrive();"):], (file, kernel)


def test_the_kernels_with_remote_stores_are_found():
    assert ("gdn.cu", "gdn_rows_kernel") in [(f, k) for f, k, _ in CASES]
