"""Dense calls whose tables go up in several slabs of depth steps (32 MB and more), from pageable memory
(staged by workers) and pinned memory, against the compact two-table path and the FP64 oracle."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import interface, migration, operators, synthetic
from oracle import oracle
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True], ids=["pageable", "pinned"])
@pytest.mark.parametrize("nz", [23, 100])
def test_dense_slabs_match_compact_path_and_oracle(pinned, nz):
    import torch
    w = synthetic.plain_medium(nx=301, nz=nz, nf=20, ns=3)
    back = operators.design_compact_table(w.nx, w.dx, w.dz, w.M, w.nk, w.dk, back=True)
    dense = [np.ascontiguousarray(operators.dense_table(t, w.omega, w.velocity, w.nextrap, dk=w.dk))
             for t in (w.table, back)]
    assert dense[0].nbytes >= 32 << 20
    if pinned:
        dense = [torch.from_numpy(t).pin_memory().numpy() for t in dense]
    shape = (w.ns, w.nf, w.nx)
    wave, shot = w.wave.reshape(shape).copy(), w.shot.reshape(shape).copy()
    img = np.zeros((w.ns, w.nz, w.nx), np.float32)
    interface.extrapolate(w.ns, w.nextrap, w.nz, w.nx, w.nf, w.nf, w.M, dense[0], dense[1], wave, shot, img)
    _, imgs, wave_c, shot_c = migration.migrate_workload(w, two_tables=True, table_back=back, image_shots=True)
    assert rel_l2(img, imgs) <= 1e-5
    assert rel_l2(wave.reshape(-1), wave_c) <= 1e-5 and rel_l2(shot.reshape(-1), shot_c) <= 1e-5
    _, so, wo, _ = oracle.migrate_workload_f64(w, tab_back=back)
    assert rel_l2(img, so) <= 1e-5 and rel_l2(wave.reshape(-1), wo) <= 1e-5
