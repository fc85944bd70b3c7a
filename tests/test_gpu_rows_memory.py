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


def test_partial_images_that_do_not_fit_run_on_fewer_ctas():
    """300 items of one CTA each would take 19.7 MB of partial images; with 12 MB half of the CTAs take two."""
    w = _survey(2, 256, 64, 300, 31)
    img, _, wave, shot = migration.migrate_workload(w)
    lib().img2d_release_host_cache()
    before = migration.Plan.for_workload(w)
    lib().img2d_release_host_cache()
    lib().img2d_set_alloc_limit(12 << 20)
    try:
        plan = migration.Plan.for_workload(w)
    finally:
        lib().img2d_set_alloc_limit(0)
    d, d0 = plan.describe(), before.describe()
    assert d["kernel"] == d0["kernel"] == "migrate_rows" and d0["grid"] * 65536 > 12 << 20 >= d["grid"] * 65536
    import torch
    dev = torch.device("cuda")
    plan.set_model(torch.from_numpy(w.omega).to(dev), torch.from_numpy(np.ascontiguousarray(w.velocity)).to(dev), w.dk,
                   torch.from_numpy(w.table).to(dev))
    wd, sd = torch.from_numpy(w.wave).to(dev), torch.from_numpy(w.shot).to(dev)
    im = torch.zeros((w.nz, w.nx), device=dev)
    plan.execute(wd, sd, im)
    np.testing.assert_array_equal(wd.cpu().numpy(), wave)
    np.testing.assert_array_equal(sd.cpu().numpy(), shot)
    assert np.linalg.norm(im.cpu().numpy() - img) <= 1e-6 * np.linalg.norm(img)
    plan.close()
    before.close()


def test_source_above_the_limit_is_not_kept():
    """Every depth step of 6 shots over 1000 x 1000 at 256 frequencies: 12.6 GB.  Keeping keeps nothing, and the
    reusing call recomputes."""
    import torch
    w = _survey(6, 1000, 1000, 256, 7)
    m = torch.from_numpy(np.random.default_rng(2).standard_normal((w.nextrap, w.nx)).astype(np.float32)).cuda()
    op = lsm.MigrationOperator.for_workload(w)
    out = []
    for mode in ("recompute", "keep", "reuse"):
        data = op.zeros_data()
        op.plan.demigrate(m, op.wave, data, source=mode)
        out.append(data.cpu().numpy())
    d = op.plan.describe_demigration()
    assert d["kernel"] == "demigrate_rows" and d["source_cache_bytes"] < 1 << 20
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2]) and float(np.abs(out[0]).max()) > 0
    op.plan.close()
    lib().img2d_release_host_cache()
