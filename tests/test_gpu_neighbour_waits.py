"""The migration kernels whose warps wait for their neighbours only, bit for bit against kernels with barriers
(the same multiply-adds per element): the 16-slot default against migrate_cluster2_kernel, the 8-slot
one against its scalar form, over their operator lengths, one to five CTAs per cluster, and launches of
many items whose windows differ."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import migration, operators, synthetic

pytestmark = pytest.mark.gpu


def _survey(ns, nx, nz, nf, taps, lo=0, seed=3):
    rng = np.random.default_rng(seed)
    v = synthetic.gaussian_random_field(nz, nx, 8.0, 1500.0, 4500.0, rng)
    x0, wn = np.zeros(ns, np.int32), np.full(ns, nx, np.int32)
    if lo:
        wn = rng.integers(lo, nx + 1, ns).astype(np.int32)
        x0 = (rng.random(ns) * (nx - wn + 1)).astype(np.int32)
    w = synthetic.Workload("waits", nz, nx, 10.0, 10.0, nf, (taps - 1) // 2, 200, 0.0, None, v, None, x0, wn,
                           (x0 + wn // 2).astype(np.int32), nextrap=nz, seed=seed)
    w = synthetic._finish(w, 2.0, 50.0, 20.0, rng, False)
    w.table = operators.design_compact_table(256, w.dx, w.dz, w.M, w.nk, w.dk)
    return w


def _equal(w, ours, other):
    img, _, wave, shot = migration.migrate_workload(w, **ours)
    img_o, _, wave_o, shot_o = migration.migrate_workload(w, **other)
    np.testing.assert_array_equal(wave, wave_o)
    np.testing.assert_array_equal(shot, shot_o)
    assert np.isfinite(wave).all() and float(np.abs(wave).max()) > 0
    assert np.linalg.norm(img - img_o) <= 1e-6 * np.linalg.norm(img_o)


@pytest.mark.parametrize("taps", [7, 9, 15, 17, 31, 33, 47, 63, 65])
@pytest.mark.parametrize("ns,nx,lo", [(16, 250, 0), (32, 512, 100), (40, 900, 200), (32, 1024, 0)])
def test_16_slots(taps, ns, nx, lo):
    w = _survey(ns, nx, 6, 2, taps, lo)
    d = migration.Plan.for_workload(w).describe()
    assert d["kernel"] == "migrate_cluster2" and d["variant"] >= 12, d  # after the variants of the table
    _equal(w, {}, dict(cluster2=True))


def test_16_slots_many_items_of_different_width():
    w = _survey(72, 475, 9, 141, 35, 59)
    d = migration.Plan.for_workload(w).describe()
    assert d["variant"] >= 12 and d["items"] > 2 * d["grid"], d
    _equal(w, {}, dict(cluster2=True))


@pytest.mark.parametrize("taps", [7, 15, 33, 65, 81])
@pytest.mark.parametrize("ns,nx,nf,lo,K", [(12, 700, 3, 0, 1), (12, 2000, 3, 300, 2), (12, 3000, 3, 0, 3), (40, 3000, 20, 300, 3),
                                           (9, 4500, 2, 0, 5)])
def test_8_slots(taps, ns, nx, nf, lo, K):
    w = _survey(ns, nx, 6, nf, taps, lo)
    d = migration.Plan.for_workload(w, wide=True).describe()
    assert d["kernel"] == "migrate_wide" and d["cluster"] in (K, K + 1), d
    _equal(w, dict(wide=True), dict(wide_scalar=True))
