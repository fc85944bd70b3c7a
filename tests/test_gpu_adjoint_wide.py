"""Wide demigration kernel at the edges of its range: 7 to 65 taps (ring from 17 on), windows of one and
several CTAs that do not fill their warps, slabs that do not divide the depth, against the FP64 oracle
(1e-5) and bit for bit against the single-CTA kernel."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import lsm, synthetic
from oracle import oracle
from tests.conftest import rel_l2
from tests.test_gpu_adjoint import _with_M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [5, 7, 9, 15, 17, 19, 33, 49, 51, 63, 65, 67])
@pytest.mark.parametrize("ns,nx,slab", [(12, 70, 3), (33, 300, 0), (17, 1300, 1)])
def test_wide_demigration(taps, ns, nx, slab):
    import torch
    w = _with_M(synthetic.plain_medium(nx=nx, nz=7, nf=2, ns=ns), (taps - 1) // 2)
    m = np.random.default_rng(1).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    ref = oracle.demigrate_workload_f64(w, m.astype(np.float64))
    out = {}
    for kw in ({}, dict(no_cluster=True)):
        op = lsm.MigrationOperator.for_workload(w, slab_depth=slab, **kw)
        modes = ("recompute", "keep", "reuse") if not kw else ("recompute",)
        for mode in modes:
            d = op.zeros_data()
            op.plan.demigrate(torch.from_numpy(m).cuda(), op.wave, d, slab_depth=slab, source=mode)
            out[mode if not kw else "single"] = d.cpu().numpy()
        if 7 <= taps <= 65 and not kw:
            op.plan.check_status()  # no wait of the wide kernel gave up
        op.plan.close()
    assert rel_l2(out["recompute"], ref) <= 1e-5
    for mode in ("keep", "reuse", "single"):
        assert np.array_equal(out[mode], out["recompute"]), mode
