"""The row-split kernel (few lane slots, table pairs): against the FP64 oracle at the compact path's bar
(relative L2 1e-5), over the operator lengths at which its tap ranges change shape, windows that do
not fill a warp's pass, more items than CTAs (partial images visited again), per-shot images, the
chunked host entry, and non-finite inputs against the general kernel."""
import numpy as np
import pytest

from imaging2d_wlsq_b200 import lsm, migration, operators, synthetic
from oracle import oracle
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _survey(ns, nx, nz, nf, taps, seed=3, gaps=False):
    """ns shots over nx positions; gaps: disjoint apertures M samples apart (they share a slot)."""
    M = (taps - 1) // 2
    rng = np.random.default_rng(seed)
    v = synthetic.gaussian_random_field(nz, nx, 8.0, 1500.0, 4500.0, rng)
    if gaps:
        wn = (nx - (ns - 1) * M) // ns
        x0 = np.arange(ns, dtype=np.int32) * (wn + M)
        wn = np.full(ns, wn, dtype=np.int32)
    else:
        x0, wn = np.zeros(ns, np.int32), np.full(ns, nx, np.int32)
    pos = (x0 + wn // 2).astype(np.int32)
    w = synthetic.Workload("rows", nz, nx, 10.0, 10.0, nf, M, 200, 0.0, None, v, None, x0.astype(np.int32), wn, pos,
                           nextrap=nz, seed=seed)
    return synthetic._finish(w, 2.0, 50.0, 20.0, rng, True)


def _kernel(w, **kw):
    return migration.Plan.for_workload(w, **kw).describe()


def _check(w, img, wave, shot, **kw):
    stack, _, wo, so = oracle.migrate_workload_f64(w, **kw)
    assert rel_l2(img, stack) <= 1e-5
    assert rel_l2(wave, wo) <= 1e-5 and rel_l2(shot, so) <= 1e-5


@pytest.mark.parametrize("taps", [3, 5, 7, 9, 15, 17, 23, 25, 31, 33, 41, 49, 57, 63, 65, 79])
@pytest.mark.parametrize("ns,nx", [(1, 33), (2, 129), (3, 200)])
def test_rows_matches_oracle(taps, ns, nx):
    w = _survey(ns, nx, 5, 3, taps)
    assert _kernel(w)["kernel"] == "migrate_rows"
    img, _, wave, shot = migration.migrate_workload(w)
    _check(w, img, wave, shot)


@pytest.mark.parametrize("taps", [7, 25, 43, 55, 73])
def test_rows_two_tables_match_general_kernel_and_oracle(taps):
    w = _survey(5, 150, 5, 4, taps)
    back = operators.design_compact_table(w.nx, w.dx, w.dz, w.M, w.nk, w.dk, back=True)
    back = (back * np.exp(0.3j)).astype(np.complex64)  # not the conjugate of the forward table
    assert _kernel(w, two_tables=True)["kernel"] == "migrate_rows"
    img, imgs, wave, shot = migration.migrate_workload(w, two_tables=True, table_back=back, image_shots=True)
    ref, refs, wave_g, shot_g = migration.migrate_workload(w, two_tables=True, table_back=back, image_shots=True,
                                                           generic=True)
    assert rel_l2(img, ref) <= 1e-5 and rel_l2(imgs, refs) <= 1e-5
    assert rel_l2(wave, wave_g) <= 1e-5 and rel_l2(shot, shot_g) <= 1e-5


def test_rows_more_items_than_ctas_and_narrow_windows():
    """24 shots, 6 to a slot, 500 frequencies: CTAs accumulate several items, whose windows do not
    cover the model, into their partial images."""
    w = _survey(24, 24 * 40 + 23 * 5, 4, 500, 11, gaps=True)
    w.shot_x0, w.shot_nx = w.shot_x0[::2].copy(), w.shot_nx[::2].copy()  # every other one: room to spare
    w.shot_pos = w.shot_pos[::2].copy()
    w = synthetic._finish(w, 2.0, 50.0, 20.0, np.random.default_rng(1), True)
    img, imgs, wave, shot = migration.migrate_workload(w, image_shots=True)
    _check(w, img, wave, shot)
    w2 = _survey(5, 96, 3, 1200, 9)
    d = _kernel(w2)
    assert d["kernel"] == "migrate_rows" and d["items"] > d["grid"], d
    img, _, wave, shot = migration.migrate_workload(w2)
    _check(w2, img, wave, shot)


def test_rows_chunked_host_entry_matches_plan():
    """A host call of 80 MB of spectra runs in frequency chunks that share two sets of partial images."""
    import torch
    w = _survey(2, 2000, 2, 2600, 7)
    assert _kernel(w)["kernel"] == "migrate_rows"
    img, _, wave, shot = migration.migrate_workload(w)
    dev = torch.device("cuda")
    plan = migration.Plan.for_workload(w)
    plan.set_model(torch.from_numpy(w.omega).to(dev), torch.from_numpy(np.ascontiguousarray(w.velocity)).to(dev),
                   w.dk, torch.from_numpy(w.table).to(dev))
    wd, sd = torch.from_numpy(w.wave.copy()).to(dev), torch.from_numpy(w.shot.copy()).to(dev)
    im = torch.zeros((w.nz, w.nx), device=dev)
    plan.execute(wd, sd, im)
    np.testing.assert_array_equal(wave, wd.cpu().numpy())
    np.testing.assert_array_equal(shot, sd.cpu().numpy())
    assert rel_l2(img, im.cpu().numpy()) <= 1e-6
    plan.close()


@pytest.mark.parametrize("taps", [7, 25, 31])
def test_rows_non_finite_inputs_reach_what_they_reach_in_the_general_kernel(taps):
    w = _survey(2, 2 * 40 + (taps - 1) // 2, 1, 2, taps, gaps=True)
    w.shot[39] = np.inf       # last sample of the first shot: M samples before the second one
    w.wave[5] = np.nan
    assert _kernel(w)["kernel"] == "migrate_rows"
    _, _, wave, shot = migration.migrate_workload(w)
    _, _, wave_g, shot_g = migration.migrate_workload(w, generic=True)
    for a, b in ((wave, wave_g), (shot, shot_g)):
        np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b))
        np.testing.assert_array_equal(np.isnan(a.real), np.isnan(b.real))
        np.testing.assert_array_equal(np.isnan(a.imag), np.isnan(b.imag))


@pytest.mark.parametrize("taps", [3, 5, 7, 9, 15, 17, 25, 31, 41, 57, 63, 65, 79])
@pytest.mark.parametrize("ns,nx", [(1, 33), (2, 130), (3, 65), (2, 1000)])
def test_rows_demigration_matches_oracle(taps, ns, nx):
    """Row-split demigration, one and two slots per item (1000 positions with long operators leave
    room for one), every source mode."""
    import torch
    w = _survey(ns, nx, 4, 3, taps)
    m = np.random.default_rng(2).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    ref = oracle.demigrate_workload_f64(w, m.astype(np.float64))
    op = lsm.MigrationOperator.for_workload(w)
    out = []
    for mode in ("recompute", "keep", "reuse"):
        d = op.zeros_data()
        op.plan.demigrate(torch.from_numpy(m).cuda(), op.wave, d, source=mode)
        out.append(d.cpu().numpy())
        assert rel_l2(out[-1], ref) <= 1e-5
    assert op.plan.describe_demigration()["kernel"] == "demigrate_rows"
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    op.plan.close()


def test_rows_demigration_with_little_memory_takes_the_slab_kernel():
    import torch
    from imaging2d_wlsq_b200._lib import lib
    w = _survey(2, 256, 64, 8, 31)
    m = np.random.default_rng(2).standard_normal((w.nextrap, w.nx)).astype(np.float32)
    ref = oracle.demigrate_workload_f64(w, m.astype(np.float64))
    op = lsm.MigrationOperator.for_workload(w)
    lib().img2d_set_alloc_limit(1 << 20)  # every S_l: 8 CTAs x 64 planes of 4 KB; checkpoints: a quarter
    try:
        d = op.demigrate(torch.from_numpy(m).cuda())
    finally:
        lib().img2d_set_alloc_limit(0)
    assert op.plan.describe_demigration()["kernel"] == "demigrate"
    assert rel_l2(d.cpu().numpy(), ref) <= 1e-5
    op.plan.close()


@pytest.mark.parametrize("ns", [1, 2])
@pytest.mark.parametrize("nz", [1, 2, 3])
def test_rows_few_depth_steps(ns, nz):
    """The last depth step looks ahead to row offsets of a step that does not exist."""
    w = _survey(ns, 300, nz, 4, 7)
    assert _kernel(w)["kernel"] == "migrate_rows"
    img, _, wave, shot = migration.migrate_workload(w)
    _check(w, img, wave, shot)
