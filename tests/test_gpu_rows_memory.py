"""The row-split kernels with little memory."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import lsm, migration
from imaging2d_wlsq_b200._lib import lib
from tests.test_gpu_rows import _survey

pytestmark = pytest.mark.gpu


def test_recomputing_call_without_memory_leaves_the_kept_source():
    """A recomputing demigration whose planes (8 CTAs x 64 of 4 KB) do not fit runs on fewer CTAs, and the
    source kept before serves the next call."""
    import torch
    w = _survey(2, 256, 64, 8, 31)
    m = torch.from_numpy(np.random.default_rng(2).standard_normal((w.nextrap, w.nx)).astype(np.float32)).cuda()
    op = lsm.MigrationOperator.for_workload(w)
    kept = op.demigrate(m).cpu().numpy()
    lib().img2d_release_host_cache()  # no block of another plan to take
    lib().img2d_set_alloc_limit(1 << 20)
    try:
        again = op.zeros_data()
        op.plan.demigrate(m, op.wave, again)
        reused = op.demigrate(m)
    finally:
        lib().img2d_set_alloc_limit(0)
    assert op.plan.describe_demigration()["kernel"] == "demigrate_rows"
    assert np.array_equal(again.cpu().numpy(), kept) and np.array_equal(reused.cpu().numpy(), kept)
    op.plan.close()


def test_partial_images_of_a_large_model_are_bounded():
    """5 narrow shots over 4096 x 1000: the partial images of several CTAs per SM would take 14.5 GB."""
    x0 = (np.arange(5) * 100).astype(np.int32)  # overlapping: a slot each
    plan = migration.Plan(5, 1000, 1000, 4096, 256, 256, 15, 100, x0, np.full(5, 600, np.int32))
    d, held = plan.describe(), plan.workspace_bytes
    plan.close()
    lib().img2d_release_host_cache()
    assert d["kernel"] == "migrate_rows"
    assert held <= (8 << 30) + 256 * 1000 * 4096 * 2 + (64 << 20)  # and the operator index
