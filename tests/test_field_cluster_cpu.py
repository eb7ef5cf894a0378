"""The order of the cluster form's start, read from the source: every block of the cluster has to run
before a block stores into another's shared memory, so field_cg_kernel meets a barrier of the
cluster before its first reduction, whose stores go to every block."""
from __future__ import annotations

import re
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "op-pic_b200" / "csrc" / "field.cu"


def test_cluster_barrier_before_the_first_remote_store():
    text = re.sub(r"//[^\n]*", "", SRC.read_text())
    assert text.count("map_shared_rank(") == 1  # the reduction's
    body = text[text.index("field_cg_kernel(const"):]
    barrier = re.search(r"if \(kCluster\) cg::this_cluster\(\)\.sync\(\);", body)
    assert barrier and barrier.start() < body.index("cg_all_sum<")
