"""The row-split kernels with little memory."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import lsm
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
