"""Cluster demigration of surveys whose lane-slot groups differ in width (FP64 oracle, 1e-5)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import synthetic
from oracle import oracle
from tests.conftest import rel_l2
from tests.test_gpu_adjoint import _op, _with_M

pytestmark = pytest.mark.gpu


def test_cluster_demigration_groups_narrower_than_the_cluster():
    """A group of narrow shots at the right end of the model beside a group of full-aperture ones: the
    clusters are sized for the wide group, so the narrow one leaves CTAs whose positions would lie
    outside the model."""
    import torch
    w = synthetic.plain_medium(nx=1133, nz=6, nf=3, ns=32)
    w.shot_nx = np.concatenate([np.full(16, 1133), np.full(16, 140)]).astype(np.int32)
    w.shot_x0 = np.concatenate([np.zeros(16), np.full(16, 1133 - 140)]).astype(np.int32)
    w.shot_pos = (w.shot_x0 + w.shot_nx // 2).astype(np.int32)
    w = synthetic._finish(w, 2.0, 40.0, 20.0, np.random.default_rng(3), True)
    m = np.random.default_rng(4).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    ref = oracle.demigrate_workload_f64(w, m.astype(np.float64))
    for taps in (31, 19):
        if taps != 2 * w.M + 1:
            w = _with_M(w, (taps - 1) // 2)
            ref = oracle.demigrate_workload_f64(w, m.astype(np.float64))
        op = _op(w)
        data = op.demigrate(torch.from_numpy(m).cuda()).cpu().numpy()
        d = op.plan.describe_demigration()
        assert d["kernel"] == "demigrate_cluster" and d["cluster"] >= 2, d
        assert rel_l2(data, ref) <= 1e-5
        op.plan.close()
