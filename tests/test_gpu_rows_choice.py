"""The default kernel of surveys for which either the row-split or the wide kernel is faster by 15% or more
(measured on a B200)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import migration

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nx,nf,taps,lo,kernel", [
    (87, 979, 145, 25, 0, "migrate_cluster2"),     # 11.0 ms for 80 depth steps, row-split 16.6
    (7, 1741, 50, 35, 0, "migrate_wide"),          # 1.47, 1.91
    (8, 3997, 73, 25, 499, "migrate_rows"),        # the wide kernel takes 1.27 times as long
    (161, 695, 27, 25, 86, "migrate_rows"),        # 1.17 times
    (43, 746, 164, 31, 93, "migrate_rows"),        # 5.50, 4.08
    (14, 266, 221, 31, 33, "migrate_rows"),        # 2.03, 0.76
])
def test_default_kernel(ns, nx, nf, taps, lo, kernel):
    x0, wn = np.zeros(ns, np.int32), np.full(ns, nx, np.int32)
    if lo:
        rng = np.random.default_rng((ns, nx, lo))
        wn = rng.integers(lo, nx + 1, ns)
        left = rng.integers(0, nx, ns) - wn // 2
        x0 = np.clip(left, 0, nx - 2).astype(np.int32)
        wn = (np.clip(left + wn, x0 + 2, nx) - x0).astype(np.int32)
    plan = migration.Plan(ns, 8, 8, nx, nf, nf, (taps - 1) // 2, 500, x0, wn)
    assert plan.describe()["kernel"] == kernel
    plan.close()
