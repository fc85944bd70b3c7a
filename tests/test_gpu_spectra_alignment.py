"""Records that start 4 bytes past an 8-byte boundary (views of a survey with an odd number of samples per
shot) through the front end's two transforms, against float64 within 2e-6 relative L2 (the bar of the
front end's other tests)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import frontend
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nf", [(499, 101), (495, 60)])  # a prime length (library transform), a composite one
@pytest.mark.parametrize("first,count", [(1, 1), (1, 3), (2, 2), (0, 4)])
def test_record_spectra_of_views(nt, nf, first, count):
    import torch
    nx = 37
    rec = np.random.default_rng(nt).standard_normal((4, nt, nx)).astype(np.float32)
    view = torch.from_numpy(rec).cuda()[first:first + count]
    assert view.is_contiguous() and view.data_ptr() % 8 == (4 if first & 1 else 0)
    got = frontend.records_to_spectra(view, nf).cpu().numpy()
    ref = np.fft.fft(rec[first:first + count].astype(np.float64), axis=1)[:, :nf].reshape(-1)
    assert rel_l2(got, ref) <= 2e-6
