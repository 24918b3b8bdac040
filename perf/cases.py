"""Performance cases: the calls a user of this package times.

listed() names them, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (param file and input tables read, the
context, page-locked host arrays for the outputs), run() is one pass through
the public entry points and returns its outputs, work() the bytes and
operations that pass cannot do without, exact() the outputs in 64 bits where
they are plain numbers.

The kinds of pass:

  field  the Gaussian density and potential of one realisation
         (create_cartesian_fields) into the caller's CUDA tensors.
  dens   the physical density of one realisation (lognormal, clipped, 2LPT)
         with its redshift-bin normalisation, into the caller's CUDA tensor.
  mock   the whole driver sequence on one realisation, as main() runs it: the
         tables go up, and catalogues, count maps, intensity maps and
         convergence maps arrive in page-locked host arrays.
  los    the sequence for sparse sources that carry line-of-sight quantities:
         lensing columns, density and velocity skewers.
  batch  many independent realisations on uneven grids, replayed over streams
         (covariance runs): the count map of each comes back.

Catalogues have as many records as the realisation has sources, so they are
returned in the host arrays that hold them, zero past the last source.
"""
import math
import shutil
import tempfile

import numpy as np
import torch

import colore_gb300 as cg
from colore_gb300 import inputs

GRIDS = (64, 96, 128, 192, 256, 384, 512)
FULL_SKY = 4.0 * math.pi * (180.0 / math.pi) ** 2  # deg^2


def listed():
    return [
        # the smallest call: tests and parameter scans on coarse grids
        dict(name="field_64", kind="field", n_grid=64, z_max=0.6),
        # a radix-3 grid, the largest size of the batched workload
        dict(name="field_384", kind="field", n_grid=384, z_max=1.2),
        # the fields of the headline configuration
        dict(name="field_1024", kind="field", n_grid=1024, z_max=1.5),
        # density grids alone (output_density): lognormal at the size of c2,
        # and 2LPT with the TSC assignment
        dict(name="dens_lognormal_512", kind="dens", n_grid=512, z_max=1.0, dens_type=0, interp=1, bias_model=2),
        dict(name="dens_2lpt_256", kind="dens", n_grid=256, z_max=1.0, dens_type=2, interp=2, bias_model=1),
        # configuration c1: one lognormal population on 128^3
        dict(name="mock_c1_128", kind="mock", config="c1", n_grid=128),
        # configuration c2: two populations, count maps at nside 256
        dict(name="mock_c2_512", kind="mock", config="c2", n_grid=512),
        # c4 on the grid its tests use: 1LPT, a 64-shell intensity map, convergence
        dict(name="mock_c4_256", kind="mock", config="c4", n_grid=256, nside_count=128, nside_imap=128,
             nside_kappa=128),
        # configuration c4, the headline: 1024^3, every output
        dict(name="mock_c4_1024", kind="mock", config="c4", n_grid=1024),
        # c5 on the grid its tests use: three populations, nside 1024 count
        # and convergence maps
        dict(name="mock_c5_512", kind="mock", config="c5", n_grid=512),
        # lensed galaxies and a sparse skewer sample on one grid
        dict(name="los_192", kind="los", n_grid=192, z_max=0.9, lens_density=20.0, skewer_density=0.4, gauss=False),
        # the batched workload at a quarter of its 48 realisations
        dict(name="batch_c3_12", kind="batch", n_real=12, z_seed=3000),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["field", "field", "dens", "mock", "mock", "maps", "maps", "los", "batch"])
    z_max = round(rng.uniform(0.3, 1.5), 3)
    if kind == "field":
        return dict(kind="field", n_grid=rng.choice(GRIDS), z_max=z_max)
    if kind == "dens":
        t = rng.choice([0, 1, 2, 3])
        return dict(kind="dens", n_grid=rng.choice(GRIDS[:6]), z_max=z_max, dens_type=t, interp=rng.choice([0, 1, 2]),
                    bias_model=rng.choice([1, 2, 3]))
    if kind == "mock":  # galaxy populations and their count map
        return dict(kind="mock", config="galaxies", n_grid=rng.choice(GRIDS), z_max=z_max,
                    dens_type=rng.choice([0, 0, 1, 3]), bias_model=rng.choice([1, 2, 3]),
                    density=round(_log_uniform(rng, 5.0, 500.0), 3), bias=round(rng.uniform(0.8, 2.5), 3),
                    nside_count=rng.choice([0, 64, 128, 256, 512]))
    if kind == "maps":  # a sparse population, intensity, convergence and ISW maps
        return dict(kind="mock", config="maps", n_grid=rng.choice(GRIDS[1:5]), z_max=z_max,
                    dens_type=rng.choice([0, 1]), bias_model=rng.choice([1, 2, 3]),
                    density=round(_log_uniform(rng, 2.0, 50.0), 3), bias=round(rng.uniform(0.8, 2.0), 3),
                    nside_count=64, nside_imap=rng.choice([32, 64, 128]), nbands=rng.randint(4, 48),
                    nside_kappa=rng.choice([64, 128, 256]), n_kappa=rng.randint(1, 8))
    if kind == "los":
        return dict(kind="los", n_grid=rng.choice(GRIDS[:5]), z_max=z_max,
                    lens_density=round(_log_uniform(rng, 2.0, 40.0), 3),
                    skewer_density=round(_log_uniform(rng, 0.05, 1.0), 3), gauss=rng.random() < 0.5)
    return dict(kind="batch", n_real=rng.randint(3, 12), z_seed=rng.randint(1, 9999))


def _pop(z_max, density, bias, **more):
    return dict(nz=("flat", 0.05, z_max), density=density, bias=bias, nside_count=0, **more)


def _specs(case, seed):
    """The run specifications (colore_gb300.inputs) of a case."""
    if case["kind"] == "batch":
        specs = inputs.batch_specs(case["n_real"], case["z_seed"])
        for i, s in enumerate(specs):
            s["seed"] = 1000 * (int(seed) + 1) + i
            s["srcs"][0]["nside_count"] = 512
        return specs
    if case["kind"] == "mock" and case["config"] in inputs.CONFIGS:
        spec = inputs.scaled(case["config"], case["n_grid"])
        spec["srcs"] = [dict(s) for s in spec["srcs"]]
        if "nside_count" in case:
            for s in spec["srcs"]:
                s["nside_count"] = case["nside_count"]
        if "nside_imap" in case:
            spec["imap"] = [dict(m, nside=case["nside_imap"]) for m in spec["imap"]]
        if "nside_kappa" in case:
            spec["kappa"] = dict(spec["kappa"], nside=case["nside_kappa"])
    else:
        zm = case["z_max"]
        spec = dict(n_grid=case["n_grid"], z_min=0.05, z_max=zm, r_smooth=2.0,
                    dens_type=case.get("dens_type", 0), bias_model=case.get("bias_model", 2))
        if case["kind"] == "dens":
            spec["lpt_interp_type"] = case["interp"]
            spec["srcs"] = [_pop(zm, 10.0, ("const", 1.5)), _pop(zm, 5.0, ("1+z",))]
        elif case["kind"] == "los":
            spec["srcs"] = [_pop(zm, case["lens_density"], ("1+z",), lensing=True),
                            _pop(zm, case["skewer_density"], ("const", 2.0), skewers=True,
                                 gaussian_skewers=case["gauss"])]
        elif case["kind"] == "mock":
            spec["srcs"] = [dict(_pop(zm, case["density"], ("const", case["bias"])),
                                 nside_count=case["nside_count"])]
            if case["config"] == "maps":
                spec["imap"] = [dict(tz=0.1, bias=("const", 1.0), z_range=(0.06, 0.98 * zm), nbands=case["nbands"],
                                     nside=case["nside_imap"])]
                k = case["n_kappa"]
                spec["kappa"] = dict(z_out=[zm * (i + 1) / k for i in range(k)], nside=case["nside_kappa"])
                spec["isw"] = dict(z_out=[0.5 * zm, zm], nside=case["nside_kappa"])
    spec["seed"] = int(seed) + 1
    return [spec]


def _params(spec):
    d = tempfile.mkdtemp(prefix="colore_perf_")
    try:
        return cg.Params(inputs.write_inputs(d, spec))
    finally:
        shutil.rmtree(d, ignore_errors=True)


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _catalogue(pop):
    """Page-locked room for a population's Src records and its count slot."""
    cap = int(1.1 * pop["density"] * FULL_SKY) + 4096
    return _pinned((cap, 9), torch.float32), _pinned((1,), torch.int64)


def prepare(case, seed):
    specs = _specs(case, seed)
    prms = [_params(s) for s in specs]
    kind = case["kind"]
    if kind == "batch":
        cmaps = [_pinned((12 * s["srcs"][0]["nside_count"] ** 2,), torch.int32) for s in specs]
        return dict(kind=kind, batch=cg.Batch(prms, nstreams=8), cmaps=cmaps)
    spec, m = specs[0], cg.Mock(prms[0])
    st = dict(kind=kind, mock=m, spec=spec)
    if kind in ("field", "dens"):
        k = 2 if kind == "field" else 1
        st["grids"] = [torch.empty(cg.grid_shape(m.n), dtype=torch.float32, device="cuda") for _ in range(k)]
        return st
    st["cats"] = {i: _catalogue(s) for i, s in enumerate(spec["srcs"])}
    st["cmaps"] = {i: _pinned((12 * s["nside_count"] ** 2,), torch.int32) for i, s in enumerate(spec["srcs"])
                   if s.get("nside_count")}
    st["imaps"] = {i: _pinned((s["nbands"], 12 * s["nside"] ** 2), torch.float32)
                   for i, s in enumerate(spec.get("imap", []))}
    st["kappa"] = None
    if "kappa" in spec:
        st["kappa"] = _pinned((m.cfg.n_kappa, 12 * spec["kappa"]["nside"] ** 2), torch.float32)
    st["isw"] = None
    if "isw" in spec:
        st["isw"] = _pinned((m.cfg.n_isw, 12 * spec["isw"]["nside"] ** 2), torch.float32)
    if kind == "los":
        st["n_skw"] = int(0.85 * spec["srcs"][1]["density"] * FULL_SKY)
    m.set_host_outputs(catalogs=st["cats"], imaps=st["imaps"], kappa=st["kappa"])
    return st


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.run()
        return [r.count_map(0, out=a) for r, a in zip(b.mocks, state["cmaps"])]
    m = state["mock"]
    if kind == "field":
        m.create_cartesian_fields()
        return [m.grid(w, out=g)[:, :, :m.n] for w, g in enumerate(state["grids"])]
    if kind == "dens":
        m.create_cartesian_fields()
        m.compute_physical_density_field()
        m.compute_density_normalization()
        dens = m.grid(0, out=state["grids"][0])[:, :, :m.n]
        return [dens, m.norm_table(0, 0)[0], m.norm_table(0, 1)[0]]
    m.upload_tables()
    m.run()
    m.sync()  # the registered host arrays are final
    out = {}
    for i, (src, n) in state["cats"].items():
        out["src%d" % i], out["n%d" % i] = src, n
    for i, a in state["cmaps"].items():
        out["cmap%d" % i] = m.count_map(i, out=a)
    for i, a in state["imaps"].items():
        out["imap%d" % i] = a
    if state["kappa"] is not None:
        out["kappa"] = state["kappa"]
    if state["isw"] is not None:
        out["isw"] = m.isw(out=state["isw"])
    if kind == "los":  # the skewers of the sources that every realisation has
        out["skewers"] = [a[:state["n_skw"]] for a in m.skewers(1)]
    return out


def work(case):
    """Grids written once, every output byte once; 2.5 operations per point
    and level of each real transform, and a few tens per cell, source, map
    sample and ray step."""
    total_b = total_f = 0.0
    for spec in _specs(case, 0):
        n3 = float(spec["n_grid"]) ** 3
        fft = 2.5 * n3 * 3.0 * math.log2(spec["n_grid"])
        t = spec["dens_type"]
        nfft = 2 + (3 if t == 1 else (10 if t == 2 else 0))
        b, f = 8.0 * n3, nfft * fft
        if case["kind"] != "field":
            f += 60.0 * n3
        if case["kind"] in ("mock", "los", "batch"):
            src = sum(s["density"] for s in spec["srcs"]) * FULL_SKY
            b += 36.0 * src  # also where it stays on the device
            f += 100.0 * src + 60.0 * n3 * len(spec["srcs"])
            for s in spec["srcs"]:
                b += 4.0 * 12 * s.get("nside_count", 0) ** 2
                los = s["density"] * FULL_SKY * 0.3 * spec["n_grid"]
                if s.get("skewers"):
                    b += 8.0 * s["density"] * FULL_SKY * (spec["n_grid"] // 2)
                    f += 100.0 * los
                if s.get("lensing"):
                    f += 100.0 * los
            for m in spec.get("imap", []):
                b += 4.0 * m["nbands"] * 12 * m["nside"] ** 2
                f += 60.0 * n3
            for g in ("kappa", "isw"):
                if g in spec:
                    npix = 12.0 * spec[g]["nside"] ** 2
                    b += 4.0 * npix * len(spec[g]["z_out"])
                    f += 60.0 * npix * (spec["n_grid"] // 2)
        total_b += b
        total_f += f
    return {"bytes": total_b, "flops": total_f}


# ---- 64-bit values ----------------------------------------------------------
STREAM_FIELD = 0x46494C44  # key word of the field's random stream
M32 = 0xFFFFFFFF


def _philox2(c0, c1, k0, k1):
    """Words 0 and 1 of Philox4x32-10 at counters (c0, c1, 0, 0), int64 tensors."""
    c2 = torch.zeros_like(c0)
    c3 = torch.zeros_like(c0)
    for _ in range(10):
        p0 = c0 * 0xD2511F53
        p1 = c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & M32) ^ c1) ^ k0, p1 & M32, (((p0 >> 32) & M32) ^ c3) ^ k1, p0 & M32
        k0 = (k0 + 0x9E3779B9) & M32
        k1 = (k1 + 0xBB67AE85) & M32
    return c0, c1


def _table(ptr, n):
    return torch.tensor(np.ctypeslib.as_array(ptr, shape=(n,)).copy(), device="cuda")


def _modes(cfg, potential):
    """The half spectrum H[kz][ky][kx] of the density or the potential."""
    n, nh = cfg.n_grid, cfg.n_grid // 2 + 1
    dk = 2.0 * math.pi / cfg.l_box
    pk = _table(cfg.pkarr, cfg.numk)
    i = torch.arange(n, device="cuda")
    kc = torch.where(2 * i <= n, i, i - n).double() * dk
    kx = (torch.arange(nh, device="cuda").double() * dk).view(1, 1, -1)
    ky = kc.view(1, -1, 1)
    h = torch.empty((n, n, nh), dtype=torch.complex128, device="cuda")
    step = max(1, (1 << 24) // (n * nh))
    for z0 in range(0, n, step):
        z1 = min(n, z0 + step)
        kz = kc[z0:z1].view(-1, 1, 1)
        k2 = (kx * kx + ky * ky + kz * kz).reshape(-1)
        k2s = torch.where(k2 > 0, k2, torch.ones_like(k2))
        lg = 0.5 * torch.log10(k2s)
        ik = ((lg - cfg.logkmin) * cfg.idlogk).long()
        j = ik.clamp(0, cfg.numk - 2)
        p = pk[j] + (lg - (cfg.logkmin + j / cfg.idlogk)) * (pk[j + 1] - pk[j]) * cfg.idlogk
        p = torch.where(ik < cfg.numk - 1, p, pk[-1] * 10.0 ** (-3.0 * (lg - cfg.logkmax)))
        p = torch.where((lg - cfg.logkmin) * cfg.idlogk < 0, pk[0] * 10.0 ** (cfg.n_scal * (lg - cfg.logkmin)), p)
        m = torch.arange(z0 * n * nh, z1 * n * nh, device="cuda", dtype=torch.int64)
        w0, w1 = _philox2(m & M32, m >> 32, cfg.seed & M32, ((cfg.seed >> 32) & M32) ^ STREAM_FIELD)
        u1 = (w0 >> 8).double() * 2.0 ** -24
        u2 = (w1 >> 8).double() * 2.0 ** -24
        a = torch.sqrt(-(p / dk ** 3) * torch.log1p(-u2))
        sm = torch.exp(-0.5 * cfg.r2_smooth * k2) if cfg.do_smoothing else torch.ones_like(k2)
        if potential:
            a = a * (-cfg.prefac_lensing / k2s) * (sm if cfg.smooth_potential else 1.0)
        else:
            a = a * sm
        a = torch.where(k2 > 0, a, torch.zeros_like(a))
        h[z0:z1] = torch.polar(a, 2.0 * math.pi * u1).view(z1 - z0, n, nh)
    return h


def _field(cfg, potential):
    """The real field: FFTW's c2r, which takes the first and last column of
    each row as real, and the factor (sqrt(2 pi) / L)^3."""
    n = cfg.n_grid
    h = _modes(cfg, potential)
    h = torch.fft.ifft(h, dim=0, norm="forward")
    h = torch.fft.ifft(h, dim=1, norm="forward")
    h[:, :, 0].imag.zero_()
    h[:, :, -1].imag.zero_()
    g = torch.fft.irfft(h, n=n, dim=2, norm="forward")
    return g.mul_((math.sqrt(2.0 * math.pi) / cfg.l_box) ** 3)


def _lognormal(cfg, g, clip):
    """exp(D (g - D sigma^2 / 2)) - 1, or max(1 + D g, 0) - 1, with the growth
    factor D at each cell's corner radius."""
    n = cfg.n_grid
    s2 = float(g.square().mean() - g.mean().square())
    r_arr, d_arr = _table(cfg.r_arr_r2z, cg.NA), _table(cfg.growth_d_arr, cg.NA)
    ax = [(torch.arange(n, device="cuda").double() * (cfg.l_box / n) - cfg.pos_obs[a]).square() for a in range(3)]
    for z0 in range(0, n, 64):
        r = torch.sqrt(ax[0].view(1, 1, -1) + ax[1].view(1, -1, 1) + ax[2][z0:z0 + 64].view(-1, 1, 1))
        i = (r * cfg.glob_idr).long().clamp(max=cg.NA - 2)
        d = d_arr[i] + (d_arr[i + 1] - d_arr[i]) * (r - r_arr[i]) * cfg.glob_idr
        d = torch.where(r <= 0, torch.ones_like(d), torch.where(r >= r_arr[-1], d_arr[-1], d))
        x = g[z0:z0 + 64]
        g[z0:z0 + 64] = (1.0 + d * x).clamp(min=0.0) - 1.0 if clip else torch.expm1(d * (x - 0.5 * d * s2))
    return g


def exact(case, seed):
    if case["kind"] == "field":
        cfg = _params(_specs(case, seed)[0]).config
        return [_field(cfg, False), _field(cfg, True)]
    if case["kind"] == "dens" and case["dens_type"] in (0, 3):
        cfg = _params(_specs(case, seed)[0]).config
        return [_lognormal(cfg, _field(cfg, False), case["dens_type"] == 3), None, None]
    return None  # catalogues, maps and particle densities: decisions of a whole sequence
