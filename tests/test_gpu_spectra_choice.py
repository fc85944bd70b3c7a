"""Record spectra of lengths with few residues and long second stages (whose sums are shared out in parts),
for few and many shots, against float64 within 2e-6 relative L2 (the bar of the front end's other
tests)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import frontend
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nf", [(1149, 23), (1553, 20), (1282, 40), (2532, 23), (3000, 64), (4800, 31), (8192, 300), (61, 1),
                                   (347, 28), (1234, 19), (2938, 97), (67, 8), (128, 3)])
@pytest.mark.parametrize("ns", [1, 12, 70])
def test_record_spectra_of_few_and_many_shots(nt, nf, ns):
    import torch
    nx = 37
    rec = torch.randn((ns, nt, nx), generator=torch.Generator("cuda").manual_seed(nt), device="cuda")
    got = frontend.records_to_spectra(rec, nf).reshape(ns, nf, nx).cpu().numpy()
    ref = np.fft.fft(rec.cpu().numpy().astype(np.float64), axis=1)[:, :nf]
    assert rel_l2(got, ref) <= 2e-6
