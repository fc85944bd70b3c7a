"""Blocks of closed plans: kept for the next plan, given back on request; the bytes a plan says it holds."""
import pytest

from imaging2d_wlsq_b200 import migration, synthetic

pytestmark = pytest.mark.gpu


def test_blocks_of_closed_plans_are_reused_and_given_back():
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    w = synthetic.plain_medium(nx=1024, nz=200, nf=64, ns=16)
    migration.Plan.for_workload(w).close()  # what the first plan of a process leaves behind
    migration.release_cached_memory()
    start = free()
    plan = migration.Plan.for_workload(w)
    held, bytes_ = start - free(), plan.workspace_bytes
    assert held >= bytes_ * 0.9 and bytes_ > 100 << 20
    plan.close()
    assert start - free() >= bytes_ * 0.9  # kept ...
    plan = migration.Plan.for_workload(w)
    assert start - free() <= held + (4 << 20)  # ... and taken again
    plan.close()
    migration.release_cached_memory()
    assert start - free() <= 4 << 20


def test_workspace_counts_the_row_split_table():
    """50000 rows of 31 taps: 12.8 MB in the plan's order and as much in the row-split kernel's."""
    plan = migration.Plan(1, 4, 4, 128, 4, 4, 15, 50000)
    assert plan.describe()["kernel"] == "migrate_rows"
    assert plan.workspace_bytes >= 2 * 50000 * 32 * 8
    plan.close()
