"""Timed cases of the migration library: what its users call, over the sizes they call it with.

A case names one entry point (`kind`) and the geometry it is called with:

  migrate   migration.Plan.execute on device-resident spectra (stacked image, optionally the images
            of the single shots), one compact operator table or a forward and a backward one
  adjoint   migration.Plan.demigrate, the source recomputed inside the call
  gradient  one gradient of least-squares migration through torch autograd (lsm.demigrate forward,
            lsm.migrate backward)
  host      migration.migrate, from and to host memory, everything uploaded by the call
  dense     interface.extrapolate, the reference's call with dense operator tables in host memory
  frontend  frontend.prepare_shots, source wavelets and record spectra

ns shots of nx-wide models, nz depth steps, nf frequencies, operators of `taps` taps, nk table rows;
`lo` > 0 gives each shot an aperture of lo..nx traces around its own position, 0 the full width.
"""
import functools
import math

import numpy as np
import torch

from imaging2d_wlsq_b200 import frontend, interface, lsm, migration, operators

VMIN, VMAX = 1500.0, 4500.0
DX = DZ = 10.0
FMIN, F_PEAK = 2.0, 20.0
DT = 0.004


def _case(name, kind, ns, nx, nz, nf, taps, nk, lo=0, tables=1, per_shot=False, fmax=40.0, nt=0):
    c = dict(kind=kind, ns=ns, nx=nx, nz=nz, nf=nf, taps=taps, nk=nk, lo=lo, tables=tables, per_shot=per_shot,
             fmax=fmax, nt=nt)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a handful of full-aperture shots over a small model: the first run of a new user, and the
        # quality check of a processing sequence
        _case("few_shots_small", "migrate", 4, 320, 200, 64, 25, 1000, fmax=30.0),
        # one record at a time over a mid-size model: interactive work, and a driver that loops over shots
        _case("one_shot", "migrate", 1, 1024, 500, 256, 31, 2000),
        # the reference's demonstration survey through the driver's flow, which hands over a forward
        # and a backward table: nine shots over an odd-sized model, 43 taps
        _case("demo_two_tables", "migrate", 9, 151, 136, 60, 43, 1600, tables=2, fmax=60.0),
        # a small survey of ragged apertures with the image of every shot kept for inspection
        _case("ragged_shot_images", "migrate", 24, 701, 121, 47, 35, 1500, lo=90, per_shot=True, fmax=50.0),
        # a survey of full-aperture shots, the plain medium configuration in full
        _case("medium_survey", "migrate", 32, 1024, 500, 256, 31, 2000),
        # production: 256 shots of uneven aperture over a 2048-wide model, a quarter of its band
        _case("uneven_survey", "migrate", 256, 2048, 1000, 128, 35, 4000, lo=256, fmax=50.0),
        # fine sampling: 64 full-aperture shots over 4096 traces with 55-tap operators, the upper depths
        _case("fine_grid_long_taps", "migrate", 64, 4096, 200, 64, 55, 8000, fmax=60.0),
        # modelling (Born data of a reflectivity) for a few shots
        _case("model_few_shots", "adjoint", 5, 500, 250, 96, 31, 1000),
        # one gradient of least-squares migration, the least-squares configuration in full
        _case("lsm_gradient", "gradient", 64, 1024, 500, 256, 31, 2000),
        # host arrays in, host arrays out: a batch job that calls the library once per survey part
        _case("host_call", "host", 16, 1024, 250, 192, 31, 2000),
        # the reference's own call with dense tables, a slab of the demonstration survey's depths
        _case("dense_dropin", "dense", 9, 151, 40, 60, 43, 1600, fmax=60.0),
        # records and source positions to spectra, ahead of every migration
        _case("records_to_spectra", "frontend", 32, 1024, 0, 256, 0, 0, nt=1500),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["migrate"] * 6 + ["adjoint", "gradient", "gradient", "host", "dense", "frontend"])
    while True:
        ns, nx, nz, nf = _log(rng, 1, 256), _log(rng, 100, 4096), _log(rng, 40, 1000), _log(rng, 16, 256)
        taps = rng.choice([19, 25, 25, 31, 31, 35, 35, 43, 47, 55])
        nk = _log(rng, 1000, 8000)
        lo = max(taps, nx // 8) if rng.random() < 0.5 and ns > 1 else 0
        fmax = rng.uniform(25.0, 60.0)
        points = ns * nx * nf * nz * (0.55 if lo else 1.0)
        if kind == "frontend":
            nt = _log(rng, max(2 * nf, 300), 3000)
            if 1 << 18 <= ns * nt * nx <= 1 << 27:
                return _case("", kind, ns, nx, 0, nf, 0, 0, nt=nt)
        elif kind == "dense":
            ns, nx, nz, nf = min(ns, 16), min(nx, 400), min(nz, 150), min(nf, 64)
            if 1 << 22 <= nz * nf * nx * taps * 8 <= 1 << 27:
                return _case("", kind, ns, nx, nz, nf, taps, nk, fmax=fmax)
        elif kind == "migrate":
            two = rng.random() < 0.2
            if 2e6 <= points <= (5e8 if two else 1.2e10) and ns * nx * nf <= 1 << 26:
                return _case("", kind, ns, nx, nz, nf, taps, nk, lo=lo, tables=2 if two else 1,
                             per_shot=ns <= 32 and rng.random() < 0.2, fmax=fmax)
        elif 2e6 <= points <= 4e9 and ns * nx * nf <= (1 << 24 if kind == "host" else 1 << 25):
            return _case("", kind, ns, nx, nz, nf, taps, nk, lo=lo, fmax=fmax)


# --------------------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _table(taps, nk, dk, back):
    """WLSQ operators for kappa[i] = i dk on a 256-point wavenumber grid (design, not data)."""
    return operators.design_compact_table(256, DX, DZ, (taps - 1) // 2, nk, dk, back=back)


def _dk(case):
    return 2.0 * math.pi * case["fmax"] / VMIN / (case["nk"] - 1)


def _omega(case):
    return 2.0 * math.pi * torch.linspace(FMIN, case["fmax"], case["nf"], dtype=torch.float64)


def _velocity(nz, nx, gen):
    """Smooth random velocity, correlation length 50 samples, clipped to [VMIN, VMAX]."""
    white = torch.randn((nz, nx), generator=gen, device="cuda", dtype=torch.float64)
    kz = torch.fft.fftfreq(nz, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    g = torch.fft.irfft2(torch.fft.rfft2(white) * torch.exp(-0.5 * (2.0 * math.pi * 25.0) ** 2 * (kz ** 2 + kx ** 2)),
                         s=(nz, nx))
    g = (g - g.mean()) / (g.std() + 1e-30)
    return (0.5 * (VMIN + VMAX) + 0.25 * (VMAX - VMIN) * g).clamp(VMIN, VMAX).contiguous()


def _apertures(case):
    """Per-shot aperture start, width and source position: the survey's geometry, the same for all its data."""
    ns, nx = case["ns"], case["nx"]
    if not case["lo"]:
        pos = np.linspace(nx / (2 * ns), nx - nx / (2 * ns), ns).astype(np.int32)
        return np.zeros(ns, np.int32), np.full(ns, nx, np.int32), pos
    rng = np.random.default_rng((case["ns"], nx, case["lo"]))
    width = rng.integers(case["lo"], nx + 1, ns)
    centre = rng.integers(0, nx, ns)
    x0 = np.clip(centre - width // 2, 0, nx - 2).astype(np.int32)
    x1 = np.clip(centre - width // 2 + width, x0 + 2, nx).astype(np.int32)
    return x0, (x1 - x0).astype(np.int32), np.clip(centre, x0, x1 - 1).astype(np.int32)


def _spectra(case, seed, wn, rel, gen):
    """Packed source spikes and receiver spectra (Ricker amplitude x complex Gaussian per trace)."""
    f = np.linspace(FMIN, case["fmax"], case["nf"])
    amp = torch.from_numpy((2.0 / math.sqrt(math.pi)) * f ** 2 / F_PEAK ** 3 * np.exp(-(f / F_PEAK) ** 2)).float().cuda()
    total = case["nf"] * int(wn.sum())
    shot = torch.randn(total, dtype=torch.complex64, device="cuda", generator=gen)
    wave = torch.zeros(total, dtype=torch.complex64, device="cuda")
    at = 0
    for n, p in zip(wn.tolist(), rel.tolist()):
        shot[at:at + case["nf"] * n].view(case["nf"], n).mul_(amp[:, None])
        wave[at:at + case["nf"] * n].view(case["nf"], n)[:, p] = amp
        at += case["nf"] * n
    return wave, shot


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d = {"omega": _omega(case).cuda(), "velocity": _velocity(case["nz"], case["nx"], gen), "dk": _dk(case)}
    d["forw"] = _table(case["taps"], case["nk"], d["dk"], False)
    d["back"] = _table(case["taps"], case["nk"], d["dk"], True) if case["tables"] == 2 or case["kind"] == "dense" else None
    d["x0"], d["wn"], pos = _apertures(case)
    d["wave"], d["shot"] = _spectra(case, seed, d["wn"], pos - d["x0"], gen)
    if case["kind"] in ("adjoint", "gradient"):
        spikes = torch.rand((case["nz"], case["nx"]), generator=gen, device="cuda") < 0.005
        r = torch.randn((1, 1, case["nz"], case["nx"]), generator=gen, device="cuda") * spikes
        k = torch.tensor([0.25, 0.5, 0.25], device="cuda")
        d["refl"] = torch.nn.functional.conv2d(r, (k[:, None] * k[None, :])[None, None], padding=1)[0, 0].contiguous()
    return d


def _plan(case, d):
    plan = migration.Plan(case["ns"], case["nz"], case["nz"], case["nx"], case["nf"], case["nf"],
                          (case["taps"] - 1) // 2, case["nk"], d["x0"], d["wn"], two_tables=case["tables"] == 2)
    dev = [None if t is None else torch.from_numpy(t).cuda() for t in (d["forw"], d["back"])]
    plan.set_model(d["omega"], d["velocity"], d["dk"], dev[0], dev[1])
    return plan


def _host(t):
    """Page-locked host copy, as a numpy array."""
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()


def _frontend_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rec = torch.randn((case["ns"], case["nt"], case["nx"]), generator=gen, device="cuda")
    return rec, np.random.default_rng(seed).integers(0, case["nx"], case["ns"])


def _dense_index(d, l, chunk=slice(None)):
    """Nearest table row of omega / v(l, x), ties to the lower row: (nf, nx) int64."""
    value = d["omega"][chunk, None] / d["velocity"][l][None, :]
    nk = d["forw"].shape[0]
    i0 = torch.floor(value / d["dk"]).clamp(0, nk - 1).long()
    best = (i0 - 1).clamp(0, nk - 1)
    dist = (best.double() * d["dk"] - value).abs()
    for o in (0, 1, 2):
        cand = (i0 + o).clamp(0, nk - 1)
        dc = (cand.double() * d["dk"] - value).abs()
        best, dist = torch.where(dc < dist, cand, best), torch.minimum(dc, dist)
    return best


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frontend":
        rec, isx = _frontend_inputs(case, seed)
        return {"case": case, "records": rec, "isx": isx}
    d = _inputs(case, seed)
    if kind == "dense":
        forw, back = (torch.from_numpy(d[k]).cuda() for k in ("forw", "back"))
        rows = torch.stack([_dense_index(d, l) for l in range(case["nz"])])
        shape = (case["ns"], case["nf"], case["nx"])
        wave, shot = (d[k].view(shape).cpu().numpy() for k in ("wave", "shot"))
        return {"case": case, "forw": forw[rows].cpu().numpy(), "back": back[rows].cpu().numpy(), "wave0": wave,
                "shot0": shot, "wave": wave.copy(), "shot": shot.copy(),
                "image": np.zeros((case["ns"], case["nz"], case["nx"]), np.float32)}
    if kind == "host":
        return {"case": case, "d": d, "omega": d["omega"].cpu().numpy(), "velocity": d["velocity"].cpu().numpy(),
                **{k + "0": _host(d[k]) for k in ("wave", "shot")}, **{k: _host(d[k]) for k in ("wave", "shot")}}
    plan = _plan(case, d)
    if kind == "migrate":
        dims = (case["nz"], case["nx"])
        return {"case": case, "d": d, "plan": plan, "wave": torch.empty_like(d["wave"]),
                "shot": torch.empty_like(d["shot"]), "image": torch.zeros(dims, device="cuda"),
                "images": torch.zeros((case["ns"], *dims), device="cuda") if case["per_shot"] else None}
    if kind == "adjoint":
        return {"case": case, "d": d, "plan": plan, "data": torch.zeros_like(d["wave"])}
    return {"case": case, "d": d, "op": lsm.MigrationOperator(plan, d["wave"])}


# --------------------------------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind, d = case["kind"], state.get("d")
    if kind == "migrate":
        # execute() leaves the final wavefields in its buffers: the spectra are kept and copied in
        state["wave"].copy_(d["wave"])
        state["shot"].copy_(d["shot"])
        state["plan"].execute(state["wave"], state["shot"], state["image"], state["images"])
        return [state["image"], state["wave"], state["shot"], state["images"]]
    if kind == "adjoint":
        state["plan"].demigrate(d["refl"], d["wave"], state["data"])
        return [state["data"]]
    if kind == "gradient":
        m = d["refl"].detach().requires_grad_(True)
        r = lsm.demigrate(m, state["op"]) - d["shot"]
        loss = 0.5 * torch.view_as_real(r).square().sum(dtype=torch.float64)
        loss.backward()
        return [r.detach(), m.grad]
    if kind == "host":
        wave, shot = state["wave"], state["shot"]
        np.copyto(wave, state["wave0"])
        np.copyto(shot, state["shot0"])
        image, _ = migration.migrate(case["ns"], case["nz"], case["nz"], case["nx"], case["nf"], case["nf"],
                                     (case["taps"] - 1) // 2, case["nk"], d["dk"], state["omega"], state["velocity"],
                                     d["forw"], wave, shot, shot_x0=d["x0"], shot_nx=d["wn"])
        return [image, wave, shot]
    if kind == "dense":
        np.copyto(state["wave"], state["wave0"])
        np.copyto(state["shot"], state["shot0"])
        interface.extrapolate(case["ns"], case["nz"], case["nz"], case["nx"], case["nf"], case["nf"],
                              (case["taps"] - 1) // 2, state["forw"], state["back"], state["wave"], state["shot"],
                              state["image"])
        return [state["image"], state["wave"], state["shot"]]
    wave, shot = frontend.prepare_shots(state["records"], state["isx"], case["nf"], 0.0, DX, DT, 0.0, DZ, VMIN)
    return [wave, shot]


def work(case):
    """Spectra, model, index source and tables read once, results written once; four real multiply-adds
    per complex tap and wavefield."""
    ns, nx, nz, nf, taps = case["ns"], case["nx"], case["nz"], case["nf"], case["taps"]
    if case["kind"] == "frontend":
        nt = case["nt"]
        return {"bytes": 4 * ns * nt * nx + 16 * ns * nf * nx, "flops": 2 * 2.5 * ns * nx * nt * math.log2(nt)}
    _, wn, _ = _apertures(case)
    samples = int(wn.sum()) * nf
    points = samples * nz
    model = 8 * nz * nx + 8 * nf + 8 * case["nk"] * taps * case["tables"]
    if case["kind"] == "dense":
        return {"bytes": 16 * nz * nf * nx * taps + 32 * samples + 4 * ns * nz * nx, "flops": points * (16 * taps + 4)}
    if case["kind"] in ("migrate", "host"):
        return {"bytes": 32 * samples + model + 4 * nz * nx * (1 + (ns if case["per_shot"] else 0)),
                "flops": points * (16 * taps + 4)}
    # modelling steps the source and the adjoint state; the gradient steps the residual as well
    if case["kind"] == "adjoint":
        return {"bytes": 16 * samples + model + 4 * nz * nx, "flops": points * (16 * taps + 4)}
    return {"bytes": 24 * samples + model + 8 * nz * nx, "flops": points * (24 * taps + 8)}


# --------------------------------------------------------------------------------------------------
# The same in 64 bits
# --------------------------------------------------------------------------------------------------

def _fir(rows, p, M, transposed=False):
    """sum_k rows[j, x, k] p[s, j, x + k - M], or the transposed sum, zero outside the model."""
    nx = p.shape[-1]
    out = torch.zeros_like(p)
    for k in range(2 * M + 1):
        o = k - M
        a, b = max(0, -o), min(nx, nx - o)
        if a >= b:
            continue
        if transposed:
            out[..., a + o:b + o].addcmul_(rows[None, :, a:b, k], p[..., a:b])
        else:
            out[..., a:b].addcmul_(rows[None, :, a:b, k], p[..., a + o:b + o])
    return out


def _unpack(packed, case, x0, wn, fs):
    """(ns, chunk, nx) complex128 of the packed per-shot blocks' frequency rows fs, zero outside the apertures."""
    out = torch.zeros((case["ns"], fs.stop - fs.start, case["nx"]), dtype=torch.complex128, device="cuda")
    at = 0
    for s, (a, n) in enumerate(zip(x0.tolist(), wn.tolist())):
        out[s, :, a:a + n] = packed[at:at + case["nf"] * n].view(case["nf"], n)[fs]
        at += case["nf"] * n
    return out


def _pack(fields, out, case, x0, wn, fs):
    at = 0
    for s, (a, n) in enumerate(zip(x0.tolist(), wn.tolist())):
        out[at:at + case["nf"] * n].view(case["nf"], n)[fs] = fields[s, :, a:a + n]
        at += case["nf"] * n


def _chunks(case, planes):
    """Frequency ranges whose `planes` complex128 wavefields take a few GB."""
    one = case["ns"] * case["nx"] * 16 * planes
    step = max(1, min(case["nf"], int(2e10 if planes > 8 else 3e9) // one))
    return [slice(a, min(case["nf"], a + step)) for a in range(0, case["nf"], step)]


def exact(case, seed):
    if case["kind"] == "frontend":
        rec, isx = _frontend_inputs(case, seed)
        t = torch.arange(case["nt"], device="cuda", dtype=torch.float64)[None, :, None] * DT
        x = DX + DX * torch.arange(case["nx"], device="cuda", dtype=torch.float64)[None, None, :]
        r = torch.sqrt(DZ ** 2 + (x - DX * torch.from_numpy(isx).cuda()[:, None, None]) ** 2)
        term = (math.pi * 30.0) ** 2 * (t - r / VMIN).float().double() ** 2  # times are single precision
        out = []
        for v in ((1.0 - 2.0 * term) * torch.exp(-term) / torch.sqrt(r), rec):
            out.append(torch.cat([torch.fft.fft(v[s].double(), dim=0)[:case["nf"]].reshape(1, -1)
                                  for s in range(case["ns"])]).reshape(-1))
        return out
    M = (case["taps"] - 1) // 2
    if case["ns"] * case["nx"] * case["nf"] * case["nz"] * case["taps"] > (4e11 if case["kind"] != "gradient" else 3e11):
        return None  # too long
    d = _inputs(case, seed)
    forw = torch.from_numpy(d["forw"]).cuda().to(torch.complex128)
    back = forw.conj().resolve_conj() if d["back"] is None else torch.from_numpy(d["back"]).cuda().to(torch.complex128)
    mask = torch.zeros((case["ns"], 1, case["nx"]), dtype=torch.complex128, device="cuda")
    for s, (a, n) in enumerate(zip(d["x0"].tolist(), d["wn"].tolist())):
        mask[s, :, a:a + n] = 1.0
    ragged = bool(case["lo"])

    def step(rows, p, transposed=False):
        p = _fir(rows, p, M, transposed)
        return p * mask if ragged else p

    args = (case, d["x0"], d["wn"])
    if case["kind"] in ("adjoint", "gradient"):
        refl = d["refl"].double()
        data = torch.zeros(d["wave"].shape, dtype=torch.complex128, device="cuda")
        grad = torch.zeros(refl.shape, dtype=torch.float64, device="cuda")
        for fs in _chunks(case, case["nz"] + 4):
            S, states = _unpack(d["wave"], *args, fs), []
            for l in range(case["nz"]):
                S = step(forw[_dense_index(d, l, fs)], S)
                states.append(S)
            V = torch.zeros_like(S)
            for l in reversed(range(case["nz"])):
                V = step(forw[_dense_index(d, l, fs)], V + refl[l] * states[l], transposed=True)
            if case["kind"] == "gradient":
                V = V - _unpack(d["shot"], *args, fs)
                R = V
                for l in range(case["nz"]):
                    R = step(back[_dense_index(d, l, fs)], R)
                    grad[l] += (states[l].real * R.real + states[l].imag * R.imag).sum(dim=(0, 1))
            _pack(V, data, *args, fs)
        return [data] if case["kind"] == "adjoint" else [data, grad]
    images = torch.zeros((case["ns"], case["nz"], case["nx"]), dtype=torch.float64, device="cuda")
    wave, shot = (torch.zeros(d["wave"].shape, dtype=torch.complex128, device="cuda") for _ in range(2))
    for fs in _chunks(case, 6):
        S, R = (_unpack(d[k], *args, fs) for k in ("wave", "shot"))
        for l in range(case["nz"]):
            at = _dense_index(d, l, fs)
            S, R = step(forw[at], S), step(back[at], R)
            images[:, l] += (S.real * R.real + S.imag * R.imag).sum(dim=1)
        _pack(S, wave, *args, fs)
        _pack(R, shot, *args, fs)
    if case["kind"] == "dense":
        shape = (case["ns"], case["nf"], case["nx"])
        return [images, wave.view(shape), shot.view(shape)]
    out = [images.sum(dim=0), wave, shot]
    return out + [images if case["per_shot"] else None] if case["kind"] == "migrate" else out
