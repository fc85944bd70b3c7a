"""The status of bounded waits: kept over later launches of the plan until it is read, read by the
solvers.  The failure is set from the host (no kernel is made to wait)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import _lib, lsm, migration, synthetic
from imaging2d_wlsq_b200._lib import LibraryError, check, lib

pytestmark = pytest.mark.gpu


def _op(ns=16):
    return lsm.MigrationOperator.for_workload(synthetic.plain_medium(nx=256, nz=6, nf=3, ns=ns), wide=True)


def _inject(plan):
    import torch
    check(lib().img2d_plan_inject_status(plan._h, 2, torch.cuda.current_stream().cuda_stream))


@pytest.mark.parametrize("ns", [2, 16])
def test_status_outlives_later_launches_and_is_cleared_by_reading(ns):
    op = _op(ns)
    with pytest.raises(LibraryError):
        op.plan.check_status()  # nothing launched yet
    d = op.demigrate(op.zeros_image())
    op.plan.check_status()
    for later in (lambda: op.migrate(d), lambda: op.demigrate(op.zeros_image())):
        _inject(op.plan)
        later()
        with pytest.raises(LibraryError, match="gave up") as e:
            op.plan.check_status()
        assert e.value.code == _lib.IMG2D_ECUDA
        op.plan.check_status()
    op.plan.close()


@pytest.mark.parametrize("solve", [lsm.lsm_cg, lsm.cgls])
def test_solvers_check(solve):
    op = _op()
    d = op.zeros_data()
    d.fill_(1.0)
    solve(op, d, 1)
    _inject(op.plan)
    with pytest.raises(LibraryError, match="gave up"):
        solve(op, d, 1)
    op.plan.close()


def test_sharded_migration_checks(monkeypatch):
    """The check after a rank's share raises what the plan reports."""
    from imaging2d_wlsq_b200 import sharding
    execute = migration.Plan.execute

    def failing(self, *a, **k):
        execute(self, *a, **k)
        _inject(self)

    w = synthetic.plain_medium(nx=256, nz=6, nf=3, ns=16)
    img = sharding.migrate_sharded(w)[0]
    assert np.isfinite(img.cpu().numpy()).all()
    monkeypatch.setattr(migration.Plan, "execute", failing)
    with pytest.raises(LibraryError, match="gave up"):
        sharding.migrate_sharded(w)
