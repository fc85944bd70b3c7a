"""Dense calls whose two tables lie in different kinds of memory: pageable, page-locked, on the device (the
copies resolve addresses of any kind)."""
import ctypes

import numpy as np
import pytest

from imaging2d_wlsq_b200._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [("pageable", "pinned"), ("pinned", "pageable"), ("pageable", "device"),
                                   ("device", "pageable")])
def test_tables_of_different_kinds(kinds):
    import torch
    ns, nz, nx, nf, M = 2, 24, 256, 16, 15  # 24 MB a table: large enough to be staged
    rng = np.random.default_rng(0)
    tab = [(rng.standard_normal((nz, nf, nx, 2 * M + 1)) + 1j * rng.standard_normal((nz, nf, nx, 2 * M + 1)))
           .astype(np.complex64) * 0.02 for _ in range(2)]
    place = {"pageable": lambda t: t, "pinned": lambda t: t.pin_memory(), "device": lambda t: t.cuda()}

    def run(kinds):
        forw, back = (place[k](torch.from_numpy(t)) for k, t in zip(kinds, tab))
        wave, shot = np.ones((ns, nf, nx), np.complex64), np.full((ns, nf, nx), 1j, np.complex64)
        img = np.zeros((ns, nz, nx), np.float32)
        fn = ctypes.CDLL(lib()._name).img2d_extrapolate_host_order
        fn.argtypes, fn.restype = [ctypes.c_int] * 7 + [ctypes.c_void_p] * 5, ctypes.c_int
        check(fn(ns, nz, nz, nx, nf, nf, M, forw.data_ptr(), back.data_ptr(), wave.ctypes.data, shot.ctypes.data,
                 img.ctypes.data))
        return img, wave, shot

    for got, ref in zip(run(kinds), run(("pageable", "pageable"))):
        assert np.isfinite(ref).all() and float(np.abs(ref).max()) > 0
        np.testing.assert_allclose(got, ref, rtol=1e-5, atol=1e-5 * float(np.abs(ref).max()))


def test_two_threads_upload_at_once():
    """One of two dense calls at a time uses the upload ring, the other plain copies; results are those of calls
    one after the other."""
    import threading
    ns, nz, nx, nf, M = 2, 24, 256, 16, 15
    rng = np.random.default_rng(1)
    tab = [[(rng.standard_normal((nz, nf, nx, 2 * M + 1)) + 1j * rng.standard_normal((nz, nf, nx, 2 * M + 1)))
            .astype(np.complex64) * 0.02 for _ in range(2)] for _ in range(2)]
    fn = ctypes.CDLL(lib()._name).img2d_extrapolate_host_order
    fn.argtypes, fn.restype = [ctypes.c_int] * 7 + [ctypes.c_void_p] * 5, ctypes.c_int

    def run(k, out):
        for i in range(3):
            wave, shot = np.ones((ns, nf, nx), np.complex64), np.full((ns, nf, nx), 1j, np.complex64)
            img = np.zeros((ns, nz, nx), np.float32)
            rc = fn(ns, nz, nz, nx, nf, nf, M, tab[k][0].ctypes.data, tab[k][1].ctypes.data, wave.ctypes.data,
                    shot.ctypes.data, img.ctypes.data)
            out[k, i] = (rc, wave, shot)

    alone, both = {}, {}
    for k in range(2):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, both)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for key, (rc, wave, shot) in alone.items():
        assert rc == both[key][0] == 0
        np.testing.assert_array_equal(both[key][1], wave)
        np.testing.assert_array_equal(both[key][2], shot)
