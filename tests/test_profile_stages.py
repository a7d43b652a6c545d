"""The step's profiled stages name what they time: the row preparation's
interval holds its kernels and nothing else, and the islands' reaches to the
solver.  Read from the order in which the step is enqueued (no GPU)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_stage_boundaries_of_the_solver():
    source = open(os.path.join(ROOT, "fyzzxyzzy-sdk_b200", "csrc", "solver.cu")).read()
    body = source[source.index("void enqueue_solver("):]
    calls = re.findall(r"hook\((kSt\w+),|\b(k_\w+)(?:<[^<>]*>)?<<<|launch\((k_\w+)|\b(for_island_solvers)\(", body)
    order = [next(x for x in c if x) for c in calls]

    def between(a, b):
        return order[order.index(a) + 1:order.index(b)]
    prep = between("kStPrep", "kStPrepJointsEnd")
    assert [x for x in prep if x.startswith("k_")] == ["k_prep_contacts", "k_prep_joints"]
    islands = between("kStIslands", "kStPgs")
    assert "k_partition_smem" in islands and "k_partition_large" in islands and "k_desc_keys" in islands
    assert "for_island_solvers" in between("kStPgs", "kStIntegrate")
