"""Workloads of the coupling step as a user's program calls them.

listed() holds the cases, draw() more of the same ranges; prepare() makes what
the caller has in hand (device inputs, plans, tables), run() is one pass
through the public entry points, work() the bytes and flops a pass cannot do
without, exact() the same outputs in 64 bits with torch alone.

Kinds:
  sht       ShtPlan.inverse_dev / forward_dev on device arrays, each precision
  wa_host   ShtPlan.xya_wa / wa_xya on host arrays in SPML's real layout: the
            call a Fortran dynamics makes, one field at a time
  ensemble  Ensemble.inverse_dev / forward_dev: members of mixed truncations
  remap     RemapPlan.apply_dev of surface fields to an ocean grid
  flux      DSFCM_Util_SfcBulkFlux_Get on device arrays
  implcpl   ImplCplPlan.forward_dev, surface values at level 1, backward_dev
  step      Step.run: transforms, remap and flux of one coupling step
Launch shapes stay at their defaults (no autotuning: it sets process-wide
knobs).
"""
import importlib
import math

import numpy as np
import torch

DEV = "cuda"
F8 = torch.float64
PREC = {"fp64": 0, "mixed": 1, "fp16": 2}  # SHT_FP64, SHT_MIXED, SHT_MIXED_FP16
# Gaussian grids (I, J) the transforms run on, with the largest truncation N
# of an alias-free quadratic grid
GRIDS = [(64, 32, 21), (96, 48, 31), (128, 64, 42), (192, 96, 63), (256, 128, 85), (384, 192, 127),
         (512, 256, 170), (768, 384, 255), (1024, 512, 341)]
LARGEST = 192 * 512 * 1024  # grid values of a batch: 48 levels x 4 fields at T341
SLOTS = {"DelVarImplCPL": 4}
OUT3 = ["WindStressX", "WindStressY", "SenHFlx", "QVapMFlx", "LatHFlx", "SfcVelTransCoef", "SfcTempTransCoef",
        "SfcQVapTransCoef", "SUwRFlx", "LUwRFlx", "SfcHFlx_ns", "SfcHFlx_sr", "DSfcHFlxDTs"]
REMAPPED = ["WindU", "WindV", "SfcAirTemp", "SfcPress", "QVap1", "LDwRFlx"]
SIG1 = (0.995, 0.01)
CONSTS = (9.8, 1004.6, 287.04, 1200.0)  # Grav, CpDry, GasRDry, DelTime


def listed():
    return [
        # One 16-level field through the drop-in for SPML at the truncation of
        # the coupled reference configuration: latency and launches.
        dict(name="wa_host_t21", kind="wa_host", N=21, I=64, J=32, batch=16, prec="fp64"),
        # The plain FP64 transforms (the default precision) of a T42L26 model.
        dict(name="sht_fp64_t42", kind="sht", N=42, I=128, J=64, batch=104, prec="fp64", dir="both"),
        # ... of a T85L32 model, and of T341L48, the largest.
        dict(name="sht_fp64_t85", kind="sht", N=85, I=256, J=128, batch=128, prec="fp64", dir="both"),
        dict(name="sht_fp64_t341", kind="sht", N=341, I=1024, J=512, batch=192, prec="fp64", dir="both"),
        # The tensor-core transforms of the same two models.
        dict(name="sht_mixed_t85", kind="sht", N=85, I=256, J=128, batch=128, prec="mixed", dir="both"),
        dict(name="sht_mixed_t341", kind="sht", N=341, I=1024, J=512, batch=192, prec="mixed", dir="both"),
        # 64 members of 16-32 levels x 4 fields, truncations T21 ... T85.
        dict(name="ensemble_mixed", kind="ensemble", b21=1500, b42=1560, b63=1470, b85=1610, prec="mixed"),
        # Six surface fields from the T85 grid to a 1-degree ocean, 30 % land.
        dict(name="remap_1deg", kind="remap", N=85, I=256, J=128, nx=360, ny=180, land=0.3, fields=6),
        # Bulk flux on the 1-degree ocean's packed column list with polar ice,
        # and on the whole 0.25-degree grid.
        dict(name="flux_1deg", kind="flux", nx=45478, ny=1, ice=True),
        dict(name="flux_quarter", kind="flux", nx=1440, ny=720, ice=False),
        # The implicit surface coupling on every T85L32 column, one tracer.
        dict(name="implcpl_t85", kind="implcpl", ncol=32768, kmax=32, ncmax=1),
        # One coupling step: T85L32 x 4 fields, 1-degree ocean, 30 % land.
        dict(name="step_t85", kind="step", N=85, I=256, J=128, batch=128, prec="mixed", nx=360, ny=180, land=0.3,
             ice=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wa_host", "sht", "sht", "sht", "ensemble", "remap", "flux", "implcpl", "step"])
    c = dict(kind=kind)
    J = 0
    if kind in ("wa_host", "sht", "step", "remap"):
        I, J, nq = rng.choice(GRIDS[:4] if kind == "wa_host" else GRIDS)
        # quadratic, linear and odd truncations of the grid
        N = rng.choice([nq, nq, nq - rng.randint(1, nq // 3), min(J - 1, nq + rng.randint(1, nq // 3))])
        c.update(N=N, I=I, J=J)
    if kind == "wa_host":
        c.update(batch=_log(rng, 1, 48), prec=rng.choice(["fp64", "fp64", "mixed"]))
    elif kind == "sht":
        c.update(batch=_log(rng, 1, min(512, LARGEST // (c["I"] * c["J"]))),
                 prec=rng.choice(["fp64", "fp64", "mixed", "fp16"]), dir=rng.choice(["inverse", "forward", "both"]))
    elif kind == "ensemble":
        c.update({"b%d" % t: _log(rng, 16, 1600) for t in (21, 42, 63, 85)},
                 prec=rng.choice(["fp64", "mixed", "fp16"]))
    elif kind == "remap":
        nx = 2 * _log(rng, 40, 720)
        c.update(nx=nx, ny=nx // 2, land=rng.choice([0.0, 0.3, 0.6]), fields=rng.randint(1, 12))
    elif kind == "flux":
        ncol = _log(rng, 500, 1440 * 720)
        ny = rng.choice([1, max(1, int(math.sqrt(ncol / 2)))])
        c.update(nx=ncol // ny, ny=ny, ice=rng.choice([True, False]))
    elif kind == "implcpl":
        kmax = rng.randint(8, 60)
        c.update(ncol=_log(rng, 500, 524288 * 16 // kmax), kmax=kmax, ncmax=rng.choice([1, 1, 2, 3]))
    else:
        nx = 2 * _log(rng, 64, 360)
        c.update(batch=_log(rng, 8, min(256, LARGEST // (c["I"] * c["J"]) // 2)),
                 prec=rng.choice(["mixed", "mixed", "fp64", "fp16"]), nx=nx, ny=nx // 2, land=rng.choice([0.0, 0.3]), ice=rng.choice([True, False]))
    if J // 2 % 16 and "prec" in c:
        c["prec"] = "fp64"  # the tensor-core plans take whole tiles of 16 latitude pairs
    return c


def _pkg():
    return importlib.import_module("dennou-ccm_gb300")


def _ncoef(N):
    return (N + 1) * (N + 2) // 2


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


# ------------------------------------------------------------------ inputs
def _nm(N):
    n = np.concatenate([np.arange(m, N + 1) for m in range(N + 1)])
    m = np.repeat(np.arange(N + 1), np.arange(N + 1, 0, -1))
    return n, m


def _spectra(N, batch, g):
    """Complex Gaussian, variance n^-3, n = 0 zero, Im = 0 for m = 0; float64 [batch, 2 ncoef]."""
    n, m = _nm(N)
    sd = np.where(n > 0, np.maximum(n, 1.0) ** -1.5, 0.0)
    w = np.stack([np.where(m == 0, sd, sd / math.sqrt(2)), np.where(m == 0, 0.0, sd / math.sqrt(2))], -1)
    x = torch.randn((batch, 2 * len(n)), dtype=F8, device=DEV, generator=g)
    return x.mul_(torch.from_numpy(w.ravel()).to(DEV))


def _axes(I, J):
    mu, w = np.polynomial.legendre.leggauss(J)
    return 2 * np.pi * np.arange(I) / I, np.arcsin(mu), np.full(I, 2 * np.pi / I), w


def _regular(nx, ny):
    e = np.deg2rad(-90 + 180 * np.arange(ny + 1) / ny)
    return ((np.arange(nx) + 0.5) * 2 * np.pi / nx, 0.5 * (e[1:] + e[:-1]), np.full(nx, 2 * np.pi / nx),
            np.sin(e[1:]) - np.sin(e[:-1]))


def _grid_fields(I, J, batch, g):
    """A temperature-like field: a zonal mean, a few waves and small-scale noise."""
    lon = torch.arange(I, dtype=F8, device=DEV) * (2 * math.pi / I)
    lat = torch.from_numpy(_axes(I, J)[1]).to(DEV)
    a = torch.randn((batch, 6), dtype=F8, device=DEV, generator=g)
    x = torch.randn((batch, J, I), dtype=F8, device=DEV, generator=g).mul_(0.3)
    x += (250 + 40 * torch.cos(lat) ** 2)[None, :, None]
    for k in range(1, 4):
        wave = a[:, 2 * k - 2, None] * torch.cos(k * lon) + a[:, 2 * k - 1, None] * torch.sin(k * lon)
        x += 5 * wave[:, None, :] * (torch.cos(lat) ** k)[None, :, None]
    return x


def _surface(nx, ny, ice, g, lat=None):
    """The bulk flux's arrays [k, ny + 2, nx + 2] (a halo of 1, interior filled) as a dict."""
    if lat is None:
        lat = torch.from_numpy(_regular(4, ny)[1]).to(DEV)[:, None].expand(ny, nx) if ny > 1 else \
            torch.asin(torch.linspace(-1, 1, nx, dtype=F8, device=DEV))[None]

    def u(lo, hi):
        return lo + (hi - lo) * torch.rand((ny, nx), dtype=F8, device=DEV, generator=g)

    def nrm(sd):
        return sd * torch.randn((ny, nx), dtype=F8, device=DEV, generator=g)

    cl = torch.cos(lat)
    sst = 273 + 27 * cl ** 2
    ta, ps = sst - 2 + u(-1, 1), 1e5 * (1 + u(-0.01, 0.01))
    wu, wv = nrm(5.0), nrm(5.0)
    q = 0.8 * 611.0 / ps * torch.exp(2425300.0 / (8.3144621 / 1.8e-2) * (1 / 273.0 - 1 / ta))
    con = torch.where(cl < 0.5, u(0, 1), torch.zeros_like(cl)) if ice else torch.zeros_like(cl)
    c1 = ps * SIG1[1] / (9.8 * 2 * 1200.0)
    z = torch.zeros_like(cl)
    rows = {"WindU": [wu], "WindV": [wv], "SfcAirTemp": [ta], "QVap1": [q], "SDwRFlx": [300 * cl.clamp_min(0)],
            "LDwRFlx": [0.8 * 5.670373e-8 * ta ** 4], "ImplCplCoef1": [c1, c1, 1616.0 * c1, c1],
            "ImplCplCoef2": [z, z, z, z], "SfcTemp": [sst, z + 271.35, z], "SfcAlbedo": [z + 0.06, z + 0.5, z],
            "SIceCon": [con], "SfcHeight": [z], "SfcPress": [ps]}
    d = {}
    for name, xs in rows.items():
        a = torch.zeros((len(xs), ny + 2, nx + 2), dtype=F8, device=DEV)
        for k, x in enumerate(xs):
            a[k, 1:-1, 1:-1] = x
        d[name] = a
    return d


def _flux_dict(d, nx, ny):
    out = dict(d)
    for n in OUT3 + ["DelVarImplCPL"]:
        out[n] = torch.zeros((SLOTS.get(n, 3), ny + 2, nx + 2), dtype=F8, device=DEV)
    out["a_Sig1Info"] = np.array(SIG1)
    return out, (nx + 2, ny + 2, 2, nx + 1, 2, ny + 1)


def _profiles(ncol, K, nc, g):
    """Atmosphere columns: half levels [K+1, ncol] (surface first), full levels [K, ncol]."""
    G, Cp, R, _ = CONSTS
    sh = 1 - (torch.arange(K + 1, dtype=F8, device=DEV)[:, None] / K) ** 1.5
    sf = 0.5 * (sh[:-1] + sh[1:])

    def u(*s):
        return torch.rand(s, dtype=F8, device=DEV, generator=g)

    def nrm(*s):
        return torch.randn(s, dtype=F8, device=DEV, generator=g)

    ps = 1e5 * (0.98 + 0.04 * u(ncol))
    ph, pf = sh * ps, sf * ps
    tf = 288 * sf ** 0.19 + 2 * u(K, ncol) - 1
    th = torch.cat([tf[:1] + 1, 0.5 * (tf[:-1] + tf[1:]), tf[-1:]])
    zf = R * tf / G * torch.log(1 / sf)
    zh = torch.cat([torch.zeros_like(zf[:1]), 0.5 * (zf[:-1] + zf[1:]), 2 * zf[-1:] - zf[-2:-1]])
    decay = torch.exp(-zh / 1000)
    kv = (10 * decay + 0.1) * (0.5 + u(ncol))
    kv[0], kv[K] = 0, 0
    top = torch.ones_like(decay)
    top[K] = 0
    f = decay * top
    q = (3e-5 + 1e-5 * nrm(nc, ncol)).abs()
    return {"MomFluxX": 0.1 * nrm(ncol) * f, "MomFluxY": 0.1 * nrm(ncol) * f, "HeatFlux": (20 + 10 * nrm(ncol)) * f,
            "QMixFlux": (q[:, None, :] * f).contiguous(), "Press": ph, "ExnerFull": (pf / 1e5) ** (R / Cp),
            "ExnerHalf": (ph / 1e5) ** (R / Cp), "VirTemp": th, "Height": zf, "VelDiffCoef": kv,
            "TempDiffCoef": 1.2 * kv, "QMixDiffCoef": 1.1 * kv}


def _level1(ncol, nc, g):
    sd = {"DUDt": 1e-3, "DVDt": 1e-3, "DTempDt": 1e-3}
    d = {k: s * torch.randn(ncol, dtype=F8, device=DEV, generator=g) for k, s in sd.items()}
    d["DQMixDt"] = 1e-7 * torch.randn((nc, ncol), dtype=F8, device=DEV, generator=g)
    return d


def _ocean(case):
    """Land mask and the indices of the ocean cells of the case's regular grid."""
    n = case["nx"] * case["ny"]
    mask = np.random.Generator(np.random.PCG64(0)).uniform(size=n) >= case["land"]
    return np.flatnonzero(mask)


def _remap_plan(case, pkg):
    S, D = _axes(case["I"], case["J"]), _regular(case["nx"], case["ny"])
    ocean = _ocean(case)
    t = pkg.gen_gridmapfile_lonlat2lonlat(S[0], S[1], D[0], D[1], S[2], S[3], D[2], D[3], weight_mode=pkg.J99_CONSERVE)
    send, recv, coef = t.index(case["I"], case["nx"])
    rank = np.full(case["nx"] * case["ny"], -1, np.int64)
    rank[ocean] = np.arange(len(ocean))
    r = rank[recv - 1]
    keep = r >= 0
    return pkg.RemapPlan(case["I"] * case["J"], len(ocean), send[keep], (r[keep] + 1).astype(np.int32), coef[keep]), len(ocean)


def _src_fields(case, fields, g):
    """Surface fields of the atmosphere grid, in the order the coupler sends them."""
    lat = torch.from_numpy(_axes(case["I"], case["J"])[1]).to(DEV)[:, None].expand(case["J"], case["I"])
    s = _surface(case["I"], case["J"], False, g, lat)
    f = [s[n][0, 1:-1, 1:-1].reshape(-1) for n in REMAPPED]
    return torch.stack([f[k % 6] * (1 + k // 6) for k in range(fields)]).contiguous()


def _seeded(case, seed):
    """The case's inputs from the seed alone (prepare and exact both start here)."""
    g, k = _gen(seed), case["kind"]
    if k == "sht":
        if case["dir"] == "forward":
            return {"grid": _grid_fields(case["I"], case["J"], case["batch"], g)}
        return {"spec": _spectra(case["N"], case["batch"], g)}
    if k == "wa_host":
        return {"spec": _spectra(case["N"], case["batch"], g)}
    if k == "ensemble":
        return {"spec": [_spectra(t, case["b%d" % t], g) for t in (21, 42, 63, 85)]}
    if k == "remap":
        return {"src": _src_fields(case, case["fields"], g)}
    if k == "flux":
        return {"sfc": _surface(case["nx"], case["ny"], case["ice"], g)}
    if k == "implcpl":
        return {"prof": _profiles(case["ncol"], case["kmax"], case["ncmax"], g),
                "lev1": _level1(case["ncol"], case["ncmax"], g)}
    n = len(_ocean(case))
    return {"spec": _spectra(case["N"], case["batch"], g), "src": _src_fields(case, 6, g),
            "sfc": _surface(n, 1, case["ice"], g)}


def _wa_index(N):
    """Positions of (Re, Im) of the m-major coefficients in SPML's real layout; -1: no Im."""
    n, m = _nm(N)
    return n * (n + 1) + m, np.where(m > 0, n * (n + 1) - m, -1)


def _to_wa(spec, N):
    re, im = _wa_index(N)
    x = spec.reshape(spec.shape[0], -1, 2)
    wa = torch.zeros((spec.shape[0], (N + 1) ** 2), dtype=F8, device=spec.device)
    wa[:, torch.from_numpy(re).to(spec.device)] = x[..., 0]
    k = np.flatnonzero(im >= 0)
    wa[:, torch.from_numpy(im[k]).to(spec.device)] = x[:, torch.from_numpy(k).to(spec.device), 1]
    return wa


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    pkg, s, k = _pkg(), _seeded(case, seed), case["kind"]
    s["case"] = case
    if k in ("sht", "wa_host", "step"):
        N, I, J, B = case["N"], case["I"], case["J"], case["batch"]
        s["plan"] = pkg.ShtPlan(N, I, J, PREC[case["prec"]], B)
        if k == "wa_host":
            s["wa"] = _to_wa(s.pop("spec"), N).cpu().numpy()
            return s
        if "grid" not in s:
            s["grid"] = torch.empty((B, J, I), dtype=F8, device=DEV)
        s["out"] = torch.empty((B, 2 * _ncoef(N)), dtype=F8, device=DEV)
    if k == "ensemble":
        dims = [(64, 32), (128, 64), (192, 96), (256, 128)]
        s["n"] = [case["b%d" % t] for t in (21, 42, 63, 85)]
        s["plan"] = pkg.Ensemble([(t, I, J, b) for t, (I, J), b in zip((21, 42, 63, 85), dims, s["n"])], PREC[case["prec"]])
        s["grid"] = [torch.empty((b, J, I), dtype=F8, device=DEV) for (I, J), b in zip(dims, s["n"])]
        s["out"] = [torch.empty_like(x) for x in s["spec"]]
    if k in ("remap", "step"):
        s["rplan"], s["ncol"] = _remap_plan(case, pkg)
    if k == "remap":
        s["dst"] = torch.empty((case["fields"], s["ncol"]), dtype=F8, device=DEV)
    if k == "flux":
        s["flux"], s["fgrid"] = _flux_dict(s.pop("sfc"), case["nx"], case["ny"])
    if k == "implcpl":
        n, K, nc = case["ncol"], case["kmax"], case["ncmax"]
        s["plan"] = pkg.ImplCplPlan(n, K, nc, 1, CONSTS)
        shapes = {"DUDt": (K, n), "DVDt": (K, n), "DTempDt": (K, n), "DQMixDt": (nc, K, n), "ImplCplCoef1": (4, n),
                  "ImplCplCoef2": (4, n)}
        s["tend"] = {a: torch.empty(v, dtype=F8, device=DEV) for a, v in shapes.items()}
    if k == "step":
        n = s["ncol"]
        d, s["fgrid"] = _flux_dict(s.pop("sfc"), n, 1)
        IA, JA = s["fgrid"][:2]
        s["remapped"] = torch.zeros((6, JA, IA), dtype=F8, device=DEV)
        d.update({name: s["remapped"][f] for f, name in enumerate(REMAPPED)})
        s["flux"] = d
        s["step"] = pkg.Step(sht=s["plan"], nfl=case["batch"], spec_in=s["spec"], grid=s["grid"], spec_out=s["out"],
                             remaps=[(s["rplan"], 6, s["src"], case["I"] * case["J"], s["remapped"].view(-1)[IA + 1:],
                                      IA * JA)], flux=d, flux_grid=s["fgrid"])
    return s


def _flux_out(f):
    return {n: f[n] for n in OUT3 + ["DelVarImplCPL", "SfcTemp", "SfcAlbedo"]}


def run(s):
    case = s["case"]
    k, st = case["kind"], torch.cuda.current_stream()
    if k == "wa_host":
        xya = s["plan"].xya_wa(s["wa"])
        return {"xya": xya, "wa": s["plan"].wa_xya(xya)}
    if k == "sht":
        out = {}
        if case["dir"] != "forward":
            s["plan"].inverse_dev(s["spec"], s["grid"], case["batch"], st)
            out["grid"] = s["grid"]
        if case["dir"] != "inverse":
            s["plan"].forward_dev(s["grid"], s["out"], case["batch"], st)
            out["spec"] = s["out"]
        return out
    if k == "ensemble":
        s["plan"].inverse_dev(s["spec"], s["grid"], s["n"], st)
        s["plan"].forward_dev(s["grid"], s["out"], s["n"], st)
        return {"grid": s["grid"], "spec": s["out"]}
    if k == "remap":
        s["rplan"].apply_dev(s["src"], case["I"] * case["J"], s["dst"], s["ncol"], case["fields"], st)
        return s["dst"]
    if k == "flux":
        _pkg().DSFCM_Util_SfcBulkFlux_Get(s["flux"], *s["fgrid"], device=True, stream=st)
        return _flux_out(s["flux"])
    if k == "implcpl":
        t = s["tend"]
        s["plan"].forward_dev(s["prof"], t, st)
        for a in ("DUDt", "DVDt", "DTempDt"):  # the coupler's surface solution
            t[a][0] = s["lev1"][a]
        t["DQMixDt"][:, 0] = s["lev1"]["DQMixDt"]
        s["plan"].backward_dev(t, st)
        return dict(t)
    s["step"].run(st)
    return {"grid": s["grid"], "spec": s["out"], "remapped": s["remapped"], **_flux_out(s["flux"])}


# ------------------------------------------------------------------- work
def _sht_work(N, I, J, B, passes):
    return (passes * 8.0 * B * (2 * _ncoef(N) + I * J),
            passes * B * (2.0 * J * _ncoef(N) + 2.5 * J * I * math.log2(I)))


def work(case):
    k = case["kind"]
    b = f = 0.0
    if k in ("sht", "wa_host", "step"):
        b, f = _sht_work(case["N"], case["I"], case["J"], case["batch"], 2 if case.get("dir", "both") == "both" else 1)
    if k == "ensemble":
        for t, (I, J) in zip((21, 42, 63, 85), [(64, 32), (128, 64), (192, 96), (256, 128)]):
            x = _sht_work(t, I, J, case["b%d" % t], 2)
            b, f = b + x[0], f + x[1]
    if k in ("remap", "step"):
        n, fields = len(_ocean(case)), case.get("fields", 6)
        nnz = n * (1 + case["I"] / case["nx"]) * (1 + case["J"] / case["ny"])  # overlaps of the two grids' cells
        b += 16 * nnz + 8.0 * fields * (case["I"] * case["J"] + n)
        f += 2 * nnz * fields
    if k in ("flux", "step"):
        n = case["nx"] * case["ny"] if k == "flux" else len(_ocean(case))
        b += 504.0 * n
        f += 315.0 * n
    if k == "implcpl":
        n, K, nc = case["ncol"], case["kmax"], case["ncmax"]
        b += 8.0 * n * ((9 + nc) * (K + 1) + (2 + 3 + nc) * K + 8)
        f += n * K * (4000.0 / 32 + (nc - 1) * 25)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ exact
def _pnm(N, J):
    """Nodes' weights and Pbar [ncoef, J] (mean square 1 over the sphere, no Condon-Shortley phase)."""
    mu, w = np.polynomial.legendre.leggauss(J)
    x, sx = torch.from_numpy(mu).to(DEV), torch.from_numpy(np.sqrt((1 - mu) * (1 + mu))).to(DEV)
    n, m = _nm(N)
    P = torch.zeros((len(n), J), dtype=F8, device=DEV)
    first = [k * (N + 1) - k * (k - 1) // 2 for k in range(N + 2)]
    pmm = torch.ones(J, dtype=F8, device=DEV)
    rows = torch.empty((N + 1, J), dtype=F8, device=DEV)
    for k in range(N + 1):
        if k:
            pmm = pmm * math.sqrt((2 * k + 1) / (2 * k)) * sx
        rows[k] = pmm
    off = torch.tensor(first[:-1], device=DEV)
    P[off] = rows
    pa, pb = torch.zeros_like(rows), rows
    mm = torch.arange(N + 1, dtype=F8, device=DEV)[:, None]
    for d in range(1, N + 1):  # n = m + d for every m at once
        c = N + 1 - d
        nn, mk = mm[:c] + d, mm[:c]
        a = torch.sqrt((4 * nn * nn - 1) / (nn * nn - mk * mk))
        bb = torch.sqrt(((nn - 1) ** 2 - mk * mk) / (4 * (nn - 1) ** 2 - 1))
        pa, pb = pb[:c], a * (x * pb[:c] - bb * pa[:c])
        P[off[:c] + d] = pb
    return torch.from_numpy(w).to(DEV), P, first


def _inverse(N, I, J, spec):
    w, P, first = _pnm(N, J)
    B = spec.shape[0]
    z = spec.reshape(B, -1, 2).permute(0, 2, 1)
    F = torch.zeros((B, J, I // 2 + 1), dtype=torch.complex128, device=DEV)
    for m in range(N + 1):
        s = slice(first[m], first[m] + N + 1 - m)
        F[:, :, m] = torch.view_as_complex((z[:, :, s] @ P[s]).permute(0, 2, 1).contiguous())
    return torch.fft.irfft(F, n=I, norm="forward")


def _forward(N, I, J, grid):
    w, P, first = _pnm(N, J)
    B = grid.shape[0]
    out = torch.empty((B, _ncoef(N), 2), dtype=F8, device=DEV)
    F = torch.empty((B, J, N + 1), dtype=torch.complex128, device=DEV)
    for b in range(0, B, 16):
        F[b:b + 16] = torch.fft.rfft(grid[b:b + 16], norm="forward")[:, :, :N + 1]
    for m in range(N + 1):
        s = slice(first[m], first[m] + N + 1 - m)
        x = torch.view_as_real(F[:, :, m].contiguous()).permute(0, 2, 1) * (0.5 * w)
        out[:, s] = (x @ P[s].T).permute(0, 2, 1)
    out[:, :N + 1, 1] = 0  # Im = 0 for m = 0
    return out.reshape(B, -1)


def _overlap(src_e, dst_e, period=None):
    """[dst, src] overlap lengths of two sets of cells given by their edges."""
    o = np.zeros((len(dst_e) - 1, len(src_e) - 1))
    for s in ([0.0] if period is None else [-period, 0.0, period]):
        lo = np.maximum(dst_e[:-1, None], src_e[None, :-1] + s)
        hi = np.minimum(dst_e[1:, None], src_e[None, 1:] + s)
        o += np.maximum(hi - lo, 0)
    return o


def _remap(case, src):
    S, D = _axes(case["I"], case["J"]), _regular(case["nx"], case["ny"])

    def lon_edges(x):
        return np.concatenate([[0.5 * (x[-1] - 2 * np.pi + x[0])], 0.5 * (x[1:] + x[:-1]), [0.5 * (x[-1] + x[0] + 2 * np.pi)]])

    def lat_edges(w):
        e = np.concatenate([[-1.0], -1 + np.cumsum(w)])
        e[-1] = 1.0
        return e

    eS, eD, xS, xD = lat_edges(S[3]), lat_edges(D[3]), lon_edges(S[0]), lon_edges(D[0])
    A = torch.from_numpy(_overlap(eS, eD) / np.diff(eD)[:, None]).to(DEV)
    B = torch.from_numpy(_overlap(xS, xD, 2 * np.pi) / np.diff(xD)[:, None]).to(DEV)
    f = A @ src.reshape(-1, case["J"], case["I"]) @ B.T
    return f.reshape(len(src), -1)[:, torch.from_numpy(_ocean(case)).to(DEV)]


def _flux(d):
    """The bulk flux in array form on the interior of the arrays d; the outputs of _flux_out."""
    R, Cp, L, StB, g, K = 8.3144621 / 1.8e-2, 1616.0, (2425300.0, 2425300.0 + 334000.0), 5.670373e-8, 9.8, 0.4
    i = {n: a[:, 1:-1, 1:-1] for n, a in d.items()}
    Ps, Ta, q1, U, V, ice = (i[n][0] for n in ("SfcPress", "SfcAirTemp", "QVap1", "WindU", "WindV", "SIceCon"))
    z = torch.zeros_like(Ps)
    ex, exs = (Ps * SIG1[0] / 1e5) ** (R / Cp), (Ps / 1e5) ** (R / Cp)
    vel = torch.sqrt(U * U + V * V)
    H, z0 = R / g * Ta * (1 - SIG1[0]), 1e-4
    cn = (K / torch.log((H + z0) / z0)) ** 2
    frac, flag = (1 - ice, ice), (torch.ones_like(ice, dtype=torch.bool), ice > 1e-12)
    v = {n: [] for n in OUT3}
    qs = []
    for n in range(2):
        Ts, al = i["SfcTemp"][n], i["SfcAlbedo"][n]
        q = 611.0 / Ps * torch.exp(L[n] / R * (1 / 273.0 - 1 / Ts))
        Ri = g / (Ts / exs) * (Ta / ex - Ts / exs) / vel.clamp_min(0.01) ** 2 * H
        rp, rn = Ri.clamp_min(0), Ri.clamp_max(0)
        s, u = torch.sqrt(1 + 5 * rp), 1 + 75 * cn * torch.sqrt(-(H + z0) / z0 * rn)
        cm = torch.where(Ri > 0, cn / (1 + 10 * rp / s), cn * (1 - 10 * rn / u)).clamp(0, 1)
        ch = torch.where(Ri > 0, cn / (1 + 15 * rp * s), cn * (1 - 15 * rn / u)).clamp(0, 1)
        w = vel.clamp(0.01, 1000) * Ps / (R * Ts)
        cm, ch = (torch.where(flag[n], x * w, z) for x in (cm, ch))
        e = -ch * (q1 - q)
        row = [-cm * U, -cm * V, -Cp * exs * ch * (Ta / ex - Ts / exs), e, L[n] * e, cm, ch, ch,
               torch.where(flag[n], al * i["SDwRFlx"][0], z), torch.where(flag[n], StB * Ts ** 4, z)]
        for name, x in zip(OUT3, row):
            v[name].append(x)
        qs.append(q)
    m = {n: frac[0] * v[n][0] + frac[1] * v[n][1] for n in OUT3[:10]}
    temp = frac[0] * i["SfcTemp"][0] ** 4 + torch.where(flag[1], frac[1] * i["SfcTemp"][1] ** 4, z)
    alb = frac[0] * i["SfcAlbedo"][0] + torch.where(flag[1], frac[1] * i["SfcAlbedo"][1], z)
    C1, C2, sf = i["ImplCplCoef1"], i["ImplCplCoef2"], Cp * exs / ex
    names = ("WindStressX", "WindStressY", "SenHFlx", "QVapMFlx")
    coef = ("SfcVelTransCoef", "SfcVelTransCoef", "SfcTempTransCoef", "SfcQVapTransCoef")
    scale = (1.0, 1.0, sf, 1.0)
    D = [(m[n] + C2[k]) / (C1[k] + scale[k] * m[coef[k]]) for k, n in enumerate(names)]
    for k, n in enumerate(names):
        for t in range(2):
            v[n][t] = v[n][t] - scale[k] * v[coef[k]][t] * D[k]
        m[n] = m[n] - scale[k] * m[coef[k]] * D[k]
    v["LatHFlx"] = [L[t] * v["QVapMFlx"][t] for t in range(2)]
    m["LatHFlx"] = frac[0] * v["LatHFlx"][0] + frac[1] * v["LatHFlx"][1]
    for t in range(2):
        Ts = i["SfcTemp"][t]
        net = v["LUwRFlx"][t] - i["LDwRFlx"][0] + v["LatHFlx"][t] + v["SenHFlx"][t]
        dfd = 4 * StB * Ts ** 3 + Cp * v["SfcTempTransCoef"][t] + \
            L[t] * v["SfcQVapTransCoef"][t] * (L[t] * qs[t] / (R * Ts ** 2))
        for name, x in (("SfcHFlx_ns", net), ("SfcHFlx_sr", v["SUwRFlx"][t] - i["SDwRFlx"][0]), ("DSfcHFlxDTs", dfd)):
            v[name].append(torch.where(flag[t], x, z))
    out = {}
    for n in OUT3:
        out[n] = torch.zeros((3,) + d["SfcPress"].shape[1:], dtype=F8, device=DEV)
        for k, x in enumerate(v[n] + ([m[n]] if n in m else [])):
            out[n][k, 1:-1, 1:-1] = x
    out["DelVarImplCPL"] = torch.zeros((4,) + d["SfcPress"].shape[1:], dtype=F8, device=DEV)
    for k in range(4):
        out["DelVarImplCPL"][k, 1:-1, 1:-1] = D[k]
    for n, x in (("SfcTemp", temp), ("SfcAlbedo", alb)):
        out[n] = d[n].clone()
        out[n][2, 1:-1, 1:-1] = x
    return out


def _tridiag(kmax, mass, tc, lo, hi, a0, a1, flux):
    """Rows of one system from the top down, eliminated; lo/hi: the couplings of level k to k-1 / k+1."""
    m0, r = [None] * (kmax + 1), [None] * (kmax + 1)
    for k in range(kmax, 0, -1):
        mm = lo[k] if k > 1 else torch.zeros_like(mass[1])
        mp = hi[k] if k < kmax else torch.zeros_like(mass[1])
        d = mass[k] + (a0[k] if k > 1 else 0) + (a1[k] if k < kmax else 0)
        b = -(flux[k] - flux[k - 1])
        if k == kmax:
            m0[k], r[k] = d / mm, b / mm
        else:
            m0[k] = (d * m0[k + 1] - mp) / (mm * m0[k + 1])
            r[k] = (b * m0[k + 1] - mp * r[k + 1]) / (mm * m0[k + 1])
    return m0, r


def _implcpl(case, p, lev1):
    G, Cp, R, dt = CONSTS
    K, nc = case["kmax"], case["ncmax"]
    P, Ef, Eh, Z = p["Press"], p["ExnerFull"], p["ExnerHalf"], p["Height"]
    mass = [None] + [-(P[k] - P[k - 1]) / G / (2 * dt) for k in range(1, K + 1)]
    geo = [None] + [P[k] / (R * p["VirTemp"][k]) / (Z[k] - Z[k - 1]) for k in range(1, K)]
    C1, C2 = torch.empty((4, case["ncol"]), dtype=F8, device=DEV), torch.empty((4, case["ncol"]), dtype=F8, device=DEV)
    out = {}

    def solve(name, coef, flux, x1, temp=False):
        tc = [None] + [p[coef][k] * geo[k] for k in range(1, K)]
        ks = range(1, K + 1)
        if temp:
            a0 = {k: Cp * Eh[k - 1] / Ef[k - 1] * tc[k - 1] for k in ks if k > 1}
            a1 = {k: Cp * Eh[k] / Ef[k - 1] * tc[k] for k in ks if k < K}
            lo = {k: -Cp * Eh[k - 1] / Ef[k - 2] * tc[k - 1] for k in ks if k > 1}
            hi = {k: -Cp * Eh[k] / Ef[k] * tc[k] for k in ks if k < K}
            ms = [None] + [Cp * x for x in mass[1:]]
        else:
            a0, a1 = {k: tc[k - 1] for k in ks if k > 1}, {k: tc[k] for k in ks if k < K}
            lo, hi = {k: -x for k, x in a0.items()}, {k: -x for k, x in a1.items()}
            ms = mass
        m0, r = _tridiag(K, ms, tc, lo, hi, a0, a1, flux)
        c1 = ms[1] + a1[1] - hi[1] / m0[2]
        c2 = -(flux[1] - flux[0]) - hi[1] * r[2] / m0[2]
        x, v = torch.empty((K, case["ncol"]), dtype=F8, device=DEV), x1
        x[0] = v / (2 * dt)
        for k in range(2, K + 1):
            v = (r[k] - v) / m0[k]
            x[k - 1] = v / (2 * dt)
        return x, c1, c2

    for a, (name, coef, flux) in enumerate([("DUDt", "VelDiffCoef", "MomFluxX"), ("DVDt", "VelDiffCoef", "MomFluxY"),
                                            ("DTempDt", "TempDiffCoef", "HeatFlux")]):
        out[name], C1[a], C2[a] = solve(name, coef, p[flux], lev1[name], a == 2)
    q = [solve("DQMixDt", "QMixDiffCoef", p["QMixFlux"][t], lev1["DQMixDt"][t]) for t in range(nc)]
    out["DQMixDt"], C1[3], C2[3] = torch.stack([x[0] for x in q]), q[0][1], q[0][2]
    out.update(ImplCplCoef1=C1, ImplCplCoef2=C2)
    return out


def exact(case, seed):
    s, k = _seeded(case, seed), case["kind"]
    if k in ("sht", "wa_host", "step"):
        dims = case["N"], case["I"], case["J"]
        grid = s.get("grid")
        grid = _inverse(*dims, s["spec"]) if grid is None else grid
    if k == "sht":
        out = {} if case["dir"] == "forward" else {"grid": grid}
        return out if case["dir"] == "inverse" else {**out, "spec": _forward(*dims, grid)}
    if k == "wa_host":
        return {"xya": grid, "wa": _to_wa(_forward(*dims, grid), case["N"])}
    if k == "ensemble":
        dims = [(21, 64, 32), (42, 128, 64), (63, 192, 96), (85, 256, 128)]
        grid = [_inverse(*d, x) for d, x in zip(dims, s["spec"])]
        return {"grid": grid, "spec": [_forward(*d, x) for d, x in zip(dims, grid)]}
    if k == "remap":
        return _remap(case, s["src"])
    if k == "flux":
        return _flux(s["sfc"])
    if k == "implcpl":
        return _implcpl(case, s["prof"], s["lev1"])
    f = _remap(case, s["src"])
    rem = torch.zeros((6,) + s["sfc"]["WindU"].shape[1:], dtype=F8, device=DEV)
    rem[:, 1, 1:-1] = f
    for j, name in enumerate(REMAPPED):
        s["sfc"][name] = rem[j:j + 1]
    return {"grid": grid, "spec": _forward(*dims, grid), "remapped": rem, **_flux(s["sfc"])}
