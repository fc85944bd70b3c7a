"""Images of the single shots from the row-split kernel where shots share a slot, against the FP64 oracle's
(relative L2 1e-5) and zero outside the apertures."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import migration
from oracle import oracle
from tests.conftest import rel_l2
from tests.test_gpu_rows import _survey

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nx,nf,taps", [(6, 6 * 40 + 5 * 5, 60, 11), (3, 3 * 61 + 2 * 15, 300, 31), (1, 90, 4, 25)])
def test_images_of_shots_that_share_a_slot(ns, nx, nf, taps):
    w = _survey(ns, nx, 4, nf, taps, gaps=True)
    assert migration.Plan.for_workload(w).describe()["kernel"] == "migrate_rows"
    img, imgs, _, _ = migration.migrate_workload(w, image_shots=True)
    stack, shots, _, _ = oracle.migrate_workload_f64(w)
    assert rel_l2(img, stack) <= 1e-5 and rel_l2(imgs, shots) <= 1e-5
    for s in range(ns):
        x0, n = int(w.shot_x0[s]), int(w.shot_nx[s])
        assert np.all(imgs[s, :, :x0] == 0) and np.all(imgs[s, :, x0 + n:] == 0)
