"""Demigration of 12 slots and more by the cluster kernel, which describe_demigration() reports under the same
name as the wide kernel ("wide" tells them apart): the lengths only it takes, and windows of about 500
positions, where its unrolled instances are the faster ones; against the FP64 oracle (relative L2
1e-5), with groups that leave CTAs of their cluster without positions, and bit for bit against the
single-CTA kernel."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import lsm, synthetic
from oracle import oracle
from tests.conftest import rel_l2
from tests.test_gpu_adjoint import _with_M

pytestmark = pytest.mark.gpu


def _survey(nx, nf, narrow, taps):
    """16 full-aperture shots and, with narrow > 0, 16 of that width at the right end of the model."""
    w = synthetic.plain_medium(nx=nx, nz=6, nf=nf, ns=32 if narrow else 16)
    if narrow:
        w.shot_nx = np.concatenate([np.full(16, nx), np.full(16, narrow)]).astype(np.int32)
        w.shot_x0 = np.concatenate([np.zeros(16), np.full(16, nx - narrow)]).astype(np.int32)
        w.shot_pos = (w.shot_x0 + w.shot_nx // 2).astype(np.int32)
        w = synthetic._finish(w, 2.0, 40.0, 20.0, np.random.default_rng(3), True)
    return w if taps == 2 * w.M + 1 else _with_M(w, (taps - 1) // 2)


@pytest.mark.parametrize("nx,nf,narrow,taps,cluster,wide", [
    (1133, 3, 140, 5, 3, False), (1133, 3, 140, 67, 3, False),
    (500, 3, 0, 25, 1, False), (490, 3, 70, 31, 1, False), (1000, 30, 140, 35, 2, False),
    (300, 3, 0, 31, 1, True), (500, 3, 0, 43, 1, True),
])
def test_cluster_kernel(nx, nf, narrow, taps, cluster, wide):
    import torch
    w = _survey(nx, nf, narrow, taps)
    m = np.random.default_rng(4).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    md = torch.from_numpy(m).cuda()
    out = {}
    for no_cluster in (False, True):
        op = lsm.MigrationOperator.for_workload(w, no_cluster=no_cluster)
        for mode in ("recompute",) if no_cluster else ("recompute", "keep", "reuse"):
            data = op.zeros_data()
            op.plan.demigrate(md, op.wave, data, source=mode)
            out[mode, no_cluster] = data.cpu().numpy()
        d = op.plan.describe_demigration()
        if not no_cluster:
            op.plan.check_status()
            assert (d["kernel"], d["cluster"], d["wide"]) == ("demigrate_cluster", cluster, wide), d
        op.plan.close()
    ref = out["recompute", False]
    assert rel_l2(ref, oracle.demigrate_workload_f64(w, m.astype(np.float64))) <= 1e-5
    for k, v in out.items():
        assert np.array_equal(v, ref), k
