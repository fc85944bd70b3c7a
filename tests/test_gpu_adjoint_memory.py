"""Demigration of 12 slots and more: the kept source takes no more memory than planes of 512 positions per
CTA would, and windows of few warps (one, a whole number, a remainder; groups of unequal width) come out
as the FP64 oracle's (relative L2 1e-5) and bit for bit alike in every source mode."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import migration, synthetic
from oracle import oracle
from tests.conftest import rel_l2
from tests.test_gpu_adjoint import _op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,narrow", [(40, 0), (64, 0), (65, 0), (300, 0), (300, 70), (512, 0), (1030, 0), (1100, 90),
                                       (1500, 0), (2100, 700)])
def test_kept_source_and_narrow_windows(nx, narrow):
    import torch
    w = synthetic.plain_medium(nx=nx, nz=11, nf=3, ns=32 if narrow else 16)
    if narrow:
        w.shot_nx = np.concatenate([np.full(16, nx), np.full(16, narrow)]).astype(np.int32)
        w.shot_x0 = np.concatenate([np.zeros(16), np.full(16, nx - narrow)]).astype(np.int32)
        w.shot_pos = (w.shot_x0 + w.shot_nx // 2).astype(np.int32)
        w = synthetic._finish(w, 2.0, 40.0, 20.0, np.random.default_rng(3), True)
    m = np.random.default_rng(4).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    migration.release_cached_memory()  # kept blocks may be up to a quarter larger than asked for
    op, md = _op(w), torch.from_numpy(m).cuda()
    out = {}
    for mode in ("recompute", "keep", "reuse"):
        data = op.zeros_data()
        op.plan.demigrate(md, op.wave, data, source=mode)
        out[mode] = data.cpu().numpy()
    op.plan.check_status()
    d = op.plan.describe_demigration()
    assert d["kernel"] == "demigrate_cluster"
    assert d["source_cache_bytes"] <= d["items"] * -(-nx // 512) * d["slabs"] * 512 * 16 * 8
    assert rel_l2(out["recompute"], oracle.demigrate_workload_f64(w, m.astype(np.float64))) <= 1e-5
    assert np.array_equal(out["keep"], out["recompute"]) and np.array_equal(out["reuse"], out["recompute"])
    op.plan.close()
