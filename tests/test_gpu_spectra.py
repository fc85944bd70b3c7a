"""Record and source spectra of lengths at which the two-stage transform changes shape (no divisor, one
of 31, odd and even halves, one and two passes of outputs, tables in and out of shared memory, 8 and
16 traces a CTA) and of the cuFFT path, against float64 transforms within 2e-6 relative L2 (the bar of
the front end's other tests)."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import frontend
from oracle import frontend_oracle as fo
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nf", [(1, 1), (2, 2), (7, 7), (16, 9), (31, 31), (62, 40), (97, 20), (300, 237),
                                   (499, 499), (1149, 23), (1500, 256), (1501, 1501), (3000, 64), (4800, 31),
                                   (8192, 300)])
@pytest.mark.parametrize("nx", [1, 37])
def test_record_spectra_lengths(nt, nf, nx):
    import torch
    rng = np.random.default_rng(nt)
    rec = rng.standard_normal((2, nt, nx)).astype(np.float32)
    x0 = np.array([0, nx // 2], np.int32)
    wn = np.array([nx, nx - nx // 2], np.int32)
    got = frontend.records_to_spectra(torch.from_numpy(rec).cuda(), nf, shot_x0=x0, shot_nx=wn).cpu().numpy()
    ref = np.concatenate([np.fft.fft(rec[s].astype(np.float64), axis=0)[:nf, x0[s]:x0[s] + wn[s]].reshape(-1)
                          for s in range(len(x0))])
    assert rel_l2(got, ref) <= 2e-6


@pytest.mark.parametrize("nt,nf,dt,fpeak", [(1500, 256, 0.004, 30.0), (200, 200, 0.004, 30.0), (301, 17, 0.001, 25.0),
                                            (64, 9, 0.02, 12.0), (700, 65, 0.0005, 8.0), (50, 20, 0.004, 0.5)])
def test_source_spectra_match_transform_of_the_wavelets(nt, nf, dt, fpeak):
    """Sources near and far (arrivals before, inside and after the record), wavelets of a few samples to
    ones longer than the record (time-domain path)."""
    nx, dx, v = 133, 12.5, 1800.0
    sx = np.array([0.0, 800.0, 9000.0])
    got = frontend.source_spectra(3, nt, nx, nf, dt, dx, dx, 10.0, v, sx, fpeak=fpeak, nt_rows=nf + 2).cpu().numpy()
    got = got.reshape(3, nf + 2, nx)
    x = dx + dx * np.arange(nx)
    r = np.sqrt(100.0 + (x[None] - sx[:, None]) ** 2)
    tau = (np.arange(nt)[None, :, None] * dt - (r / v)[:, None, :]).astype(np.float32).astype(np.float64)
    term = (np.pi * fpeak * tau) ** 2
    ref = np.fft.fft((1.0 - 2.0 * term) * np.exp(-term) / np.sqrt(r)[:, None, :], axis=1)[:, :nf]
    assert rel_l2(got[:, :nf], ref) <= 2e-6
    assert np.all(got[:, nf:] == 0)


def test_record_spectra_of_many_full_width_records():
    """A call large enough for the library transform, checked on its first and last record."""
    import torch
    ns, nt, nx, nf = 128, 1024, 2048, 512
    rec = torch.randn((ns, nt, nx), generator=torch.Generator("cuda").manual_seed(5), device="cuda")
    got = frontend.records_to_spectra(rec, nf).reshape(ns, nf, nx)
    for s in (0, ns - 1):
        ref = np.fft.fft(rec[s].cpu().numpy().astype(np.float64), axis=0)[:nf]
        assert rel_l2(got[s].cpu().numpy(), ref) <= 2e-6
