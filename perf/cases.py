"""Workloads of the analysis library, from its smallest call to its largest.

Each case is one pass through the public entry points, as a cycling assimilation
program makes it, over seeded synthetic inputs of the repository's own kinds:

  ring       drivers.l96_letkf: one Lorenz-96 analysis, FP64 or mixed
  globe      drivers.speedy_letkf: das_letkf on a SPEEDY-type lat/lon grid, FP64
  sweep      sweep.Sweep.run: the resident grid loop of a regional domain, mixed
             form (k <= 64 and k <= 128) or FP64 plain form
  core       core.core_batch_mixed and core.update_mixed on packed local rows
  largek     the large-ensemble core over index lists (BF16 storage) or packed
             FP32 rows, and its update
  relax      core.update_relax_f64 (RTPS / RTPP with relax_beta and the q clip)
  obs_space  core.obs_analysis and core.efso

Interface: listed(), draw(rng), prepare(case, seed), run(state), work(case),
exact(case, seed).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from letkf_gb300 import core as K
from letkf_gb300 import drivers as D
from letkf_gb300 import synthetic as S
from letkf_gb300.sweep import PREC_F64, PREC_MIXED, Sweep

CUT2 = float(np.float32(13.33333333))  # squared cut-off of the SCALE search, a single-precision literal there
OBS_PER_COLUMN = 15.26                 # 1e6 observations on a 256 x 256 grid


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the classic Lorenz-96 experiment: one tiny analysis, called thousands of times in a cycling run
        dict(name="ring_40_f64", kind="ring", nx=40, ne=20, precision="f64"),
        # a long ring, the mixed form over many points with short local lists
        dict(name="ring_100k_mixed", kind="ring", nx=100_000, ne=32, precision="mixed"),
        # the T30 SPEEDY analysis: 3-D u, v, t, q and 2-D fields, uneven radiosonde stations, FP64
        dict(name="globe_t30_f64", kind="globe", nlon=96, nlat=48, ne=40, nstations=600, sigma_km=500.0),
        # the regional analysis at the benchmark's density and column length, k = 64: a quarter of its area
        dict(name="regional_k64", kind="sweep", nlon=128, nlat=128, nlev=40, ne=64, nv=6, precision="mixed",
             density=1.0),
        # a serving domain with a small ensemble
        dict(name="regional_k20", kind="sweep", nlon=128, nlat=128, nlev=20, ne=20, nv=2, precision="mixed",
             density=1.0),
        # a domain with a large on-chip ensemble (the 128-wide tensor-core sweep)
        dict(name="regional_k128", kind="sweep", nlon=48, nlat=48, nlev=20, ne=128, nv=2, precision="mixed",
             density=1.0),
        # the plain form, run to check a configuration or where FP64 is asked for
        dict(name="regional_f64", kind="sweep", nlon=24, nlat=24, nlev=15, ne=64, nv=6, precision="f64",
             density=1.0),
        # a driver with its own loop: batched mixed core on packed rows, an ensemble that is no multiple of 4
        dict(name="core_k50_mixed", kind="core", npts=4001, ne=50, lmax=400, nv=5),
        # large ensembles, local lists of a few hundred, BF16 storage
        dict(name="largek_512_bf16", kind="largek", npts=256, ne=512, lmean=464, storage="bf16", spread=1.4, nv=6),
        # the same ensemble with a very wide localisation: every point needs the FP64 pass
        dict(name="largek_512_wide", kind="largek", npts=4, ne=512, lmean=24_000, storage="bf16", spread=10.0, nv=6),
        # covariance relaxation of the SCALE driver: eleven variables, spread relaxation, tapered boundary
        dict(name="relax_rtps_k50", kind="relax", npts=20_000, ne=50, nv=11, mode=K.RELAX_RTPS),
        # the analysis at observation locations and the observation sensitivity of the GFS driver
        dict(name="obs_space_k64", kind="obs_space", nloc=20_000, npts=30_000, nobs=60_000, ne=64, nlocal=50, nv=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ring", "globe", "sweep_mixed", "sweep_mixed", "sweep_f64", "core", "largek", "relax",
                       "obs_space"])
    if kind == "ring":
        precision = rng.choice(["f64", "mixed"])
        return dict(kind="ring", nx=_log_int(rng, 40, 8000 if precision == "f64" else 100_000),
                    ne=rng.randint(8, 48), precision=precision)
    if kind == "globe":
        nlon = rng.choice([48, 64, 72, 96])
        return dict(kind="globe", nlon=nlon, nlat=nlon // 2, ne=rng.randint(10, 40),
                    nstations=_log_int(rng, 100, 600), sigma_km=rng.uniform(300.0, 500.0))
    if kind == "sweep_mixed":
        ne = rng.choice([rng.randint(10, 32), rng.randint(33, 64), rng.randint(65, 128)])
        top = 128 if ne <= 64 else 56
        return dict(kind="sweep", nlon=_log_int(rng, 12, top), nlat=_log_int(rng, 12, top), nlev=rng.randint(3, 40),
                    ne=ne, nv=rng.randint(1, 6), precision="mixed", density=rng.uniform(0.2, 1.0))
    if kind == "sweep_f64":
        return dict(kind="sweep", nlon=_log_int(rng, 8, 24), nlat=_log_int(rng, 8, 24), nlev=rng.randint(3, 15),
                    ne=rng.randint(10, 64), nv=rng.randint(1, 6), precision="f64", density=rng.uniform(0.2, 1.0))
    if kind == "core":
        return dict(kind="core", npts=_log_int(rng, 100, 4000), ne=rng.randint(10, 128), lmax=_log_int(rng, 30, 400),
                    nv=rng.randint(1, 8))
    if kind == "largek":
        return dict(kind="largek", npts=_log_int(rng, 8, 256), ne=rng.randint(129, 512),
                    lmean=_log_int(rng, 100, 500), storage=rng.choice(["fp32", "bf16"]),
                    spread=rng.uniform(0.7, 2.0), nv=rng.randint(1, 8))
    if kind == "relax":
        return dict(kind="relax", npts=_log_int(rng, 1000, 20_000), ne=rng.randint(10, 100), nv=rng.randint(1, 11),
                    mode=rng.choice([K.RELAX_NONE, K.RELAX_RTPP, K.RELAX_RTPS]))
    return dict(kind="obs_space", nloc=_log_int(rng, 1000, 20_000), npts=_log_int(rng, 1000, 30_000),
                nobs=_log_int(rng, 5000, 60_000), ne=rng.randint(10, 96), nlocal=rng.randint(10, 80),
                nv=rng.randint(1, 8))


# --------------------------------------------------------------------- inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed):
    return torch.Generator(device=_dev()).manual_seed(int(seed) * 7919 + 13)


def _randn(g, *shape, dtype=torch.float64):
    return torch.randn(shape, generator=g, device=_dev(), dtype=dtype)


def _rand(g, *shape, dtype=torch.float64):
    return torch.rand(shape, generator=g, device=_dev(), dtype=dtype)


class _Modes:
    """Members as smooth random fields: per variable a few random wave vectors,
    each member its own cosine and sine coefficients."""

    def __init__(self, g, nmem, nvar, nmode, scale):
        self.k = _randn(g, nvar, nmode, 3) * scale
        self.c = _randn(g, nvar, 2 * nmode, nmem) / math.sqrt(2.0 * nmode)  # variance 1/2, as synthetic.SmoothFields

    def at(self, xyz, v):
        arg = xyz @ self.k[v].T
        return torch.cat([torch.cos(arg), torch.sin(arg)], -1) @ self.c[v]


def _ring_inputs(case, seed):
    g = _gen(seed)
    nx, ne = case["nx"], case["ne"]
    truth = 8.0 + 3.0 * torch.sin(torch.arange(nx, device=_dev(), dtype=torch.float64) * 0.7) + _randn(g, nx)
    xf = truth[:, None] + _randn(g, nx, 1) * 0.5 + _randn(g, nx, ne)
    y = truth + _randn(g, nx)
    return xf, y


def _globe_inputs(case, seed):
    c = S.speedy_case(seed, case["ne"], case["nstations"], case["nlon"], case["nlat"],
                      sigma_obs=case["sigma_km"] * 1.0e3)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())
    perm, grd = D.speedy_sort_obs(c["lon"], c["lat"], c["olon"], c["olat"], device=_dev())
    o = {k: t(c[n][perm]) for k, n in (("elm", "elm"), ("lon", "olon"), ("lat", "olat"), ("lev", "olev"),
                                      ("dat", "odat"), ("err", "oerr"))}
    gen = _gen(seed)
    nij = case["nlon"] * case["nlat"]
    g2 = torch.stack([1.0e5 + 300.0 * _randn(gen, case["ne"], nij), _rand(gen, case["ne"], nij)])
    return dict(grid={"lon": t(c["lon"]), "lat": t(c["lat"]), "nobsgrd": torch.as_tensor(grd, device=_dev())}, obs=o,
                hdxf=t(c["hdxf"][perm]), dep=t(c["dep"][perm]), gues3d=t(c["gues3d"]), gues2d=g2,
                logpfm=t(c["logpfm"]), dlon_zero=t(c["dlon_zero"]),
                params=(c["dist_zero"], c["dist_zerov"], c["dlat_zero"], c["sigma_obs"], c["sigma_obsv"]),
                var_local=np.ones((6, 7)),
                infl3d=1.05 + 0.1 * _rand(gen, 4, c["nlev"], nij), infl2d=1.05 + 0.1 * _rand(gen, 2, nij))


def _sweep_nobs(case):
    return max(64, int(case["nlon"] * case["nlat"] * OBS_PER_COLUMN * case["density"]))


def _sweep_inputs(case, seed):
    """The regional workload: clustered observations, smooth members, every
    size from the case.  Points are level-major, observations in input order."""
    rng = np.random.default_rng(seed)
    nlon, nlat, nlev, ne, nv = case["nlon"], case["nlat"], case["nlev"], case["ne"], case["nv"]
    nobs = _sweep_nobs(case)
    ri, rj, lev, cls = S.regional_obs(rng, nobs, nlon, nlat)
    err = np.where(cls == 1, 100.0, 1.0)
    g = _gen(seed)
    dx, lc = 3000.0, 60.0e3
    f = _Modes(g, ne + 1, nv, 6, 1.0)
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_dev())
    lnp = np.where(cls == 1, math.log(S.REGIONAL_P_BOT), np.log(lev))
    xyz = torch.stack([t(ri) * dx / lc, t(rj) * dx / lc, t(lnp) / 0.8], -1)
    var = torch.as_tensor(rng.integers(0, nv, nobs), device=_dev())
    hx = torch.empty((nobs, ne + 1), dtype=torch.float64, device=_dev())
    for v in range(nv):
        hx[var == v] = f.at(xyz[var == v], v)
    mem = hx[:, :ne].float().double()
    mean = mem.mean(1, keepdim=True)
    hdxf = (mem - mean).float()
    y = hx[:, ne] + t(err) * _randn(g, nobs)
    dep = (y - mean[:, 0]).cpu().numpy()
    dat = np.where(cls == 1, 1.0e5 * (1 + 0.01 * rng.standard_normal(nobs)), y.cpu().numpy())
    nij = nlon * nlat
    jj, ii = np.divmod(np.arange(nij), nlon)
    plev = S.regional_levels(nlev)
    pri, prj = np.tile(ii + 1.0, nlev), np.tile(jj + 1.0, nlev)
    prlev = np.repeat(plev, nij)
    xb = torch.empty((nv, nij * nlev, ne), dtype=torch.float32, device=_dev())
    gx, gy = t(ii + 1.0) * dx / lc, t(jj + 1.0) * dx / lc
    for l in range(nlev):
        at = torch.stack([gx, gy, torch.full_like(gx, math.log(plev[l]) / 0.8)], -1)
        for v in range(nv):
            xb[v, l * nij:(l + 1) * nij] = f.at(at, v)[:, :ne].float()
    infl = 1.0 + 0.1 * _rand(g, nij * nlev)
    prm = S.scale_params(dict(dx=dx, dy=dx, sigma_obs=S.REGIONAL_SIGMA_OBS, sigma_obsv=S.REGIONAL_SIGMA_OBSV))
    return dict(ri=ri, rj=rj, lev=lev, cls=cls, err=err, dep=dep, dat=dat, hdxf=hdxf, pri=pri, prj=prj, prlev=prlev,
                xb=xb, infl=infl, params=prm)


def _core_inputs(case, seed):
    g = _gen(seed)
    n, ne, lmax = case["npts"], case["ne"], case["lmax"]
    cnt = (_rand(g, n).square() * (lmax + 1)).long().clamp(max=lmax)  # many short lists, some empty, a few long
    offs = torch.zeros(n + 1, dtype=torch.int64, device=_dev())
    offs[1:] = cnt.cumsum(0)
    nr = int(offs[-1])
    # a row mixes a few directions shared by all points (correlated observations) with its own
    rows = _randn(g, nr, 24) @ _randn(g, 24, ne) / math.sqrt(24.0) + 0.3 * _randn(g, nr, ne)
    rows = (rows - rows.mean(1, keepdim=True)).float()
    rl = torch.exp(-6.0 * _rand(g, nr)).float()
    rd = (0.5 + _rand(g, nr)).float() / rl
    dep = _randn(g, nr).float()
    infl = 1.0 + 0.2 * _rand(g, n)
    xb = (10.0 * _randn(g, case["nv"], n, 1) + _randn(g, case["nv"], n, ne)).float()
    return dict(offs=offs, rows=rows, rl=rl, rd=rd, dep=dep, infl=infl, xb=xb)


def _largek_inputs(case, seed):
    g = _gen(seed)
    n, ne, lm = case["npts"], case["ne"], case["lmean"]
    cnt = ((0.5 + _rand(g, n)) * lm).long().clamp(min=1)
    offs = torch.zeros(n + 1, dtype=torch.int64, device=_dev())
    offs[1:] = cnt.cumsum(0)
    nr = int(offs[-1])
    nobs = int(max(2.0 * lm, 20_000))
    pos = torch.sort(_rand(g, nobs)).values * nobs / 400.0  # a line of observations; each list a stretch of it
    xyz = torch.stack([pos, _randn(g, nobs), _randn(g, nobs)], -1)
    f = _Modes(g, ne, 4, 24, 0.5)
    kind = (_rand(g, nobs) * 4).long().clamp(max=3)
    hx = torch.empty((nobs, ne), dtype=torch.float64, device=_dev())
    for v in range(4):
        hx[kind == v] = case["spread"] * f.at(xyz[kind == v], v)
    ens = hx - hx.mean(1, keepdim=True)
    ens = ens.bfloat16() if case["storage"] == "bf16" else ens.float()
    start = (_rand(g, n) * (nobs - cnt + 1)).long()
    point = torch.repeat_interleave(torch.arange(n, device=_dev()), cnt)
    within = torch.arange(nr, device=_dev()) - offs[point]
    idx = (start[point] + within).int()
    z = (within.double() / cnt[point].double() - 0.5) * 5.0
    rl = torch.exp(-0.5 * z * z).float()
    rd = torch.ones(nr, dtype=torch.float32, device=_dev())
    dep = (_randn(g, nobs) * math.sqrt(1.0 + 0.5 * case["spread"] ** 2)).float()
    infl = 1.0 + 0.1 * _rand(g, n)
    mean = 10.0 * _randn(g, case["nv"], n)
    pert = _randn(g, case["nv"], n, ne)
    pert = pert - pert.mean(-1, keepdim=True)
    return dict(offs=offs, idx=idx, ens=ens, rl=rl, rd=rd, dep=dep, infl=infl, mean=mean.float(),
                pert=pert.bfloat16() if case["storage"] == "bf16" else pert.float())


def _relax_inputs(case, seed):
    g = _gen(seed)
    n, ne, nv = case["npts"], case["ne"], case["nv"]
    w = _randn(g, n, ne, ne) * (0.1 / math.sqrt(ne))
    w = 0.5 * (w + w.transpose(1, 2)) + 0.8 * torch.eye(ne, dtype=torch.float64, device=_dev())
    pao = torch.bmm(w, w) / (ne - 1)
    tm = 0.1 * _randn(g, n, ne)
    xb = 5.0 + _randn(g, nv, n, 1) + _randn(g, nv, n, ne)
    ri, rj = 1 + 200 * _rand(g, n), 1 + 250 * _rand(g, n)
    rlev = 1e4 + 9e4 * _rand(g, n)
    return dict(w=w, pao=pao, tm=tm, xb=xb, ri=ri, rj=rj, rlev=rlev)


def _obs_space_inputs(case, seed):
    g = _gen(seed)
    n, ne, npts, nobs, nv, nl = (case[k] for k in ("nloc", "ne", "npts", "nobs", "nv", "nlocal"))
    trans = _randn(g, n, ne, ne) * (0.1 / math.sqrt(ne)) + 0.8 * torch.eye(ne, dtype=torch.float64, device=_dev())
    hdxf = _randn(g, n, ne)
    hdxf = hdxf - hdxf.mean(1, keepdim=True)
    ybar = 5.0 + _randn(g, n)
    mode = (_rand(g, n) * 3).int()
    cnt = (2.0 * nl * _rand(g, npts)).long()
    offs = torch.zeros(npts + 1, dtype=torch.int64, device=_dev())
    offs[1:] = cnt.cumsum(0)
    nr = int(offs[-1])
    # neighbouring points share observations, as a local search gives them
    point = torch.repeat_interleave(torch.arange(npts, device=_dev()), cnt)
    span = max(4 * nl, 64)
    idx = ((point.double() / npts * max(nobs - span, 1)).long() + (_rand(g, nr) * span).long()).clamp(max=nobs - 1)
    key = torch.sort(point * nobs + idx).values
    idx = (key % nobs).int()
    return dict(trans=trans, hdxf=hdxf, ybar=ybar, mode=mode, offs=offs, idx=idx, rd=0.5 + _rand(g, nr),
                rl=_rand(g, nr), hdxa=_randn(g, nobs, ne), fcst=_randn(g, nv, npts, ne), fcer=_randn(g, nv, npts),
                obsdep=_randn(g, nobs), term=[v % 3 if v < 5 else -1 for v in range(nv)])


# ------------------------------------------------------------ prepare and run
class _HandleBuffer:
    """A device buffer of a sweep handle for torch; keeps the handle alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3)


@functools.lru_cache(maxsize=None)
def _analysis_stream():
    return torch.cuda.Stream()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "ring":
        xf, y = _ring_inputs(case, seed)
        st.update(xf=xf, hxf=xf.clone(), y=y,
                  cell=torch.arange(1, case["nx"] + 1, dtype=torch.int32, device=_dev()))
    elif kind == "globe":
        st.update(_globe_inputs(case, seed))
    elif kind == "sweep":
        p = _sweep_inputs(case, seed)
        f64 = case["precision"] == "f64"
        n, ne, nv = p["pri"].size, case["ne"], case["nv"]
        sw = Sweep(ne, nv, case["nlon"], case["nlat"], n, p["params"], precision=PREC_F64 if f64 else PREC_MIXED)
        sw.set_points(p["pri"], p["prj"], p["prlev"])
        hdxf, xb = (p["hdxf"].double(), p["xb"].double()) if f64 else (p["hdxf"], p["xb"])
        sw.set_obs(p["ri"], p["rj"], p["lev"], p["dat"], p["err"], p["dep"], p["cls"], hdxf.cpu().numpy())
        sw.set_background_device(xb.data_ptr())
        _, xa, infl, nobsl = sw.device_buffers()
        at = lambda ptr, shape, t: torch.as_tensor(_HandleBuffer(sw, ptr, shape, t), device=_dev())
        st.update(sweep=sw, infl0=p["infl"], stream=_analysis_stream(), xa=at(xa, (nv, n, ne), "<f8" if f64 else "<f4"),
                  infl=at(infl, (n,), "<f8"), nobsl=at(nobsl, (n,), "<i4"))
    elif kind == "core":
        st.update(_core_inputs(case, seed))
    elif kind == "largek":
        p = _largek_inputs(case, seed)
        if case["storage"] == "fp32":
            p["rows"], p["rdep"] = K.gather_rows(p["idx"], p["ens"], p["dep"])
            p["xb"] = p["mean"][..., None] + p["pert"]
        st.update(p)
    elif kind == "relax":
        st.update(_relax_inputs(case, seed))
    else:
        st.update(_obs_space_inputs(case, seed))
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "ring":
        xa, _ = D.l96_letkf(st["xf"], st["hxf"], st["y"], st["cell"], precision=case["precision"])
        return {"xa": xa}
    if kind == "globe":
        i3, i2 = st["infl3d"].clone(), st["infl2d"].clone()
        a3, a2 = D.speedy_letkf(st["grid"], st["obs"], st["hdxf"], st["dep"], st["gues3d"], st["logpfm"],
                                st["dlon_zero"], st["params"], st["var_local"], i3, st["gues2d"], i2)
        return {"anal3d": a3, "anal2d": a2, "infl3d": i3, "infl2d": i2}
    if kind == "sweep":
        # every cycle starts from the given inflation field
        with torch.cuda.stream(st["stream"]):
            st["infl"].copy_(st["infl0"])
        st["sweep"].run(stream=st["stream"].cuda_stream)
        return {"xa": st["xa"], "infl": st["infl"], "nobsl": st["nobsl"]}
    if kind == "core":
        infl = st["infl"].clone()
        o = K.core_batch_mixed(case["ne"], st["offs"], st["rows"], st["rd"], st["rl"], st["dep"], infl,
                               want_transm=True, rdiag_wloc=True)
        xa = K.update_mixed(st["xb"], o["trans"], o["transm"])
        return {"trans": o["trans"], "transm": o["transm"], "infl": infl, "status": o["status"], "xa": xa}
    if kind == "largek":
        infl = st["infl"].clone()
        if case["storage"] == "bf16":
            o = K.core_batch_largek_indexed(case["ne"], st["offs"], st["idx"], st["ens"], st["dep"], st["rd"],
                                            st["rl"], infl, want_transm=True)
            mean, pert = K.update_bf16(st["mean"], st["pert"], o["trans"], o["transm"])
            xa = {"mean": mean, "pert": pert}
        else:
            o = K.core_batch_largek(case["ne"], st["offs"], st["rows"], st["rd"], st["rl"], st["rdep"], infl,
                                    want_transm=True)
            xa = {"xa": K.update_mixed(st["xb"], o["trans"], o["transm"])}
        return {"trans": o["trans"], "transm": o["transm"], "infl": infl, "status": o["status"], **xa}
    if kind == "relax":
        beta = K.relax_beta(st["ri"], st["rj"], st["rlev"], case["nv"], 1, 1, 3e4, 30e3, 3e3, 3e3, 200, 250, 2, 2)
        rtps = case["mode"] == K.RELAX_RTPS
        xa, infl = K.update_relax_f64(st["xb"], st["w"], st["tm"], st["pao"] if rtps else None, mode=case["mode"],
                                      alpha=0.0 if case["mode"] == K.RELAX_NONE else 0.9, beta=beta, q_var=0,
                                      q_sprd_max=0.15)
        return {"beta": beta, "xa": xa, "infl": infl} if rtps else {"beta": beta, "xa": xa}
    anal, mean = K.obs_analysis(st["trans"], st["ybar"], st["hdxf"], 0.5, st["mode"], 0.1)
    djdy, sense = K.efso(case["ne"], st["offs"], st["idx"], st["rd"], st["rl"], st["hdxa"], st["fcst"], st["fcer"],
                         st["term"], st["obsdep"])
    return {"anal": anal, "mean": mean, "djdy": djdy, "sense": sense}


# ----------------------------------------------------------------------- work
def _core_flops(ne, local):
    """One point: symmetric Gram, departure product, symmetric eigendecomposition
    (or what stands for it), W and wbar."""
    return local * ne * (ne + 1.0) + 2.0 * local * ne + 9.0 * ne ** 3 + 2.0 * ne ** 3 + 4.0 * ne ** 2


def _sweep_local(case):
    """Mean local observations of a point: the cut-off ellipsoid's share of a
    full-depth cylinder is 0.63 at these vertical scales, the domain's edges
    take a little off."""
    r = math.sqrt(CUT2) * S.REGIONAL_SIGMA_OBS / 3000.0
    edge = 1.0
    for n in (case["nlon"], case["nlat"]):
        edge *= 1.0 - min(0.5, 0.42 * r / n)
    return 0.63 * math.pi * r * r * OBS_PER_COLUMN * case["density"] * edge


def work(case):
    kind, ne = case["kind"], case["ne"]
    if kind == "ring":
        n, local = case["nx"], min(21, case["nx"])
        return {"bytes": n * (3.0 * ne + 1) * 8, "flops": n * (_core_flops(ne, local) + 2.0 * ne * ne)}
    if kind == "globe":
        nij = case["nlon"] * case["nlat"]
        n, nobs = 7 * nij, 26.2 * case["nstations"]
        # share of the sphere inside the horizontal cut-off, stations clustered; a vertical window of about 0.3
        cap = 0.5 * (1.0 - math.cos(math.sqrt(40.0 / 3.0) * case["sigma_km"] / 6371.3))
        local = nobs * cap * 0.3
        return {"bytes": 2.0 * 8 * ne * (4 * n + 2 * nij) + nobs * (ne + 7) * 8,
                "flops": n * _core_flops(ne, local) + 2.0 * ne * ne * (4 * n + 2 * nij)}
    if kind == "sweep":
        e = 8 if case["precision"] == "f64" else 4
        n, nobs = case["nlon"] * case["nlat"] * case["nlev"], _sweep_nobs(case)
        return {"bytes": 2.0 * n * case["nv"] * ne * e + nobs * (ne * e + 48.0) + n * 20.0,
                "flops": n * (_core_flops(ne, _sweep_local(case)) + 2.0 * case["nv"] * ne * ne)}
    if kind == "core":
        n, local = case["npts"], case["lmax"] / 3.0
        return {"bytes": n * (local * (ne + 3.0) * 4 + ne * (ne + 1.0) * 4 * 2 + 2.0 * case["nv"] * ne * 4),
                "flops": n * (_core_flops(ne, local) + 2.0 * case["nv"] * ne * ne)}
    if kind == "largek":
        e = 2 if case["storage"] == "bf16" else 4
        n, local, nv = case["npts"], case["lmean"], case["nv"]
        nobs = max(2.0 * local, 20_000) if case["storage"] == "bf16" else n * local
        return {"bytes": min(nobs, n * local) * (ne * e + 4.0) + n * local * 12.0 + n * ne * (ne + 1.0) * 4 * 2
                + 2.0 * n * nv * ne * e,
                "flops": n * (_core_flops(ne, local) + 2.0 * nv * ne * ne)}
    if kind == "relax":
        n, nv = case["npts"], case["nv"]
        mats = 2 if case["mode"] == K.RELAX_RTPS else 1
        return {"bytes": 8.0 * n * (mats * ne * ne + ne + 2.0 * nv * ne + nv), "flops": 2.0 * mats * n * nv * ne * ne}
    n, npts, nv = case["nloc"], case["npts"], case["nv"]
    nt = min(3, nv)
    return {"bytes": 8.0 * (n * (ne * ne * 2 / 3 + 2.0 * ne + 2) + npts * nv * (ne + 1.0) + case["nobs"] * (ne + 7.0))
            + npts * case["nlocal"] * 20.0,
            "flops": n * 2.0 * ne * ne * 2 / 3 + npts * (2.0 * nv * ne + case["nlocal"] * 2.0 * ne * nt)}


# ---------------------------------------------------------------- 64-bit values
def _inv_sqrt(a):
    """(A)^(-1/2) of a batch of symmetric positive definite matrices: coupled
    Newton iteration from the Frobenius norm, then steps anchored to A."""
    n = a.shape[-1]
    eye = torch.eye(n, dtype=a.dtype, device=a.device)
    s = a.flatten(1).norm(dim=1)[:, None, None]
    y, z = a / s, eye.expand_as(a).clone()
    for _ in range(60):
        t = torch.bmm(z, y)
        r = float((t - eye).flatten(1).norm(dim=1).max())
        t = 1.5 * eye - 0.5 * t
        y, z = torch.bmm(y, t), torch.bmm(t, z)
        if r < 1.0e-4:
            break
    z = 0.5 * (z + z.transpose(1, 2))
    for _ in range(2):
        q = torch.bmm(z, torch.bmm(a / s, z))
        z = 1.5 * z - 0.5 * torch.bmm(q, z)
        z = 0.5 * (z + z.transpose(1, 2))
    return z / s.sqrt()


def _analysis(ne, gram, b, p1, p3, some, infl):
    """W = T, wbar and the adaptive inflation of a batch of points (FP64);
    some: the points that have observations."""
    eye = torch.eye(ne, dtype=gram.dtype, device=gram.device)
    z = _inv_sqrt(gram + ((ne - 1) / infl)[:, None, None] * eye)
    w = torch.where(some[:, None, None], math.sqrt(ne - 1.0) * z, infl.sqrt()[:, None, None] * eye)
    wbar = torch.where(some[:, None], torch.bmm(z, torch.bmm(z, b[..., None]))[..., 0], torch.zeros_like(b))
    q2 = gram.diagonal(dim1=1, dim2=2).sum(1) / (ne - 1)
    q4 = (p1 - p3) / q2 - infl
    so = 2.0 / p3 * ((infl * q2 + p3) / q2) ** 2
    return w, wbar, torch.where(some, infl + 0.0016 / (so + 0.0016) * q4, infl)


def _weighted(w, rows):
    """sum_o w[p, o] y_o y_o^T for every point p."""
    ne = rows.shape[1]
    return (w @ (rows[:, :, None] * rows[:, None, :]).flatten(1)).reshape(-1, ne, ne)


def _updated(xb, w, wbar):
    """xb [nv, p, k] -> mean + x' (W + wbar 1^T)."""
    m = xb.mean(-1, keepdim=True)
    x = xb - m
    return m + torch.einsum("vpk,pkm->vpm", x, w) + torch.einsum("vpk,pk->vp", x, wbar)[..., None]


def _exact_ring(case, seed):
    xf, y = _ring_inputs(case, seed)
    nx, ne = xf.shape
    mean = xf.mean(1, keepdim=True)
    hd, dep = xf - mean, y - mean[:, 0]
    off = torch.arange(-(nx // 2), nx - nx // 2, device=_dev())
    off = off[off.abs().double() < 6.0 * math.sqrt(10.0 / 3.0)]
    r = torch.exp(-0.5 * (off.double() / 3.0) ** 2)
    off, r = off[r >= 1.0e-4], r[r >= 1.0e-4]
    out = torch.empty_like(xf)
    for p in torch.arange(nx, device=_dev()).split(20_000):
        at = (p[:, None] + off) % nx
        rows, d = hd[at], dep[at]
        gram = torch.einsum("plk,l,plm->pkm", rows, r, rows)
        b = torch.einsum("plk,l,pl->pk", rows, r, d)
        one = torch.ones(p.numel(), dtype=torch.float64, device=_dev())
        w, wbar, _ = _analysis(ne, gram, b, (d * d) @ r, r.sum() * one, one > 0, 1.05 * one)
        out[p] = _updated(xf[p][None], w, wbar)[0]
    return {"xa": out}


def _exact_globe(case, seed):
    p = _globe_inputs(case, seed)
    o, lon, lat = p["obs"], p["grid"]["lon"], p["grid"]["lat"]
    nlon, nlat = case["nlon"], case["nlat"]
    dz, dzv, dlat, so, sov = p["params"]
    # band and cell of an observation; the box of a point, with the wrap of the search
    below = lambda x, axis, lim: torch.searchsorted(axis[1:lim + 1].contiguous(), x.contiguous(), right=True) + 1
    band, cell = below(o["lat"], lat, nlat - 1), below(o["lon"], lon, nlon - 1)
    glon, glat = lon.repeat(nlat), lat.repeat_interleave(nlon)
    lo, hi = glon - p["dlon_zero"], glon + p["dlon_zero"]
    whole = hi - lo >= 360.0
    lo, hi = torch.where(whole, 0.0 * lo, lo), torch.where(whole, 0.0 * hi + 360.0, hi)
    jmin, jmax = below(glat - dlat, lat, nlat - 2), below(glat + dlat, lat, nlat - 2)
    wl, wr = lo < 0, hi > 360.0
    lo, hi = torch.where(wl, lo + 360.0, lo), torch.where(wr, hi - 360.0, hi)
    imin, imax = below(lo, lon, nlon - 1), below(hi, lon, nlon - 1)
    rad = lambda x: x * 3.1415926535 / 180.0
    ps = o["elm"] == S.ID_PS
    nij, nlev = nlon * nlat, p["logpfm"].shape[0]
    ne = case["ne"]
    yy = (p["hdxf"][:, :, None] * p["hdxf"][:, None, :]).flatten(1)
    rinv = 1.0 / o["err"] ** 2
    g3 = p["gues3d"].permute(0, 1, 3, 2)  # [nv, nlev, nij, ne]
    a3, i3 = torch.empty_like(g3), torch.empty_like(p["infl3d"])
    a2 = torch.empty_like(p["gues2d"].permute(0, 2, 1))
    for q in torch.arange(nij, device=_dev()).split(1024):
        c = cell[None, :]
        one = wl[q] ^ wr[q]
        plain, both = ~wl[q] & ~wr[q], wl[q] & wr[q]
        a, b = imin[q][:, None], imax[q][:, None]
        box = ((c >= a) & (c <= b)).double()
        full = torch.ones_like(box)
        split = (c <= b).double() + (c >= a).double()
        over = torch.where(wr[q], imax[q] > imin[q], imin[q] < imax[q])
        times = torch.where((plain | (both & (imin[q] <= imax[q])))[:, None], box,
                            torch.where((one & ~over)[:, None], split, full))
        times = times * ((band[None] >= jmin[q][:, None]) & (band[None] <= jmax[q][:, None]))
        cosd = (torch.sin(rad(o["lat"]))[None] * torch.sin(rad(glat[q]))[:, None]
                + torch.cos(rad(o["lat"]))[None] * torch.cos(rad(glat[q]))[:, None]
                * torch.cos(rad(glon[q])[:, None] - rad(o["lon"])[None]))
        dist = torch.acos(cosd.clamp(-1.0, 1.0)) * 6371.3e3
        times = times * (dist <= dz)
        for l in range(nlev):
            lev = (torch.log(torch.where(ps, o["dat"], o["lev"]))[None] - p["logpfm"][l, q][:, None]).abs()
            if l == 0:
                lev = torch.where(ps[None], torch.zeros_like(lev), lev)
            times_l = times * (lev <= dzv)
            rloc = torch.exp(-0.5 * ((dist / so) ** 2 + (lev / sov) ** 2)) * times_l
            w = rloc * rinv
            gram = (w @ yy).reshape(-1, ne, ne)
            t, wbar, infl = _analysis(ne, gram, (w * p["dep"]) @ p["hdxf"], w @ p["dep"] ** 2, rloc.sum(1),
                                      times_l.sum(1) > 0, p["infl3d"][0, l, q])
            i3[:, l, q] = infl
            a3[:, l, q] = _updated(g3[:, l, q], t, wbar)
            if l >= 4:
                a3[3, l, q] = g3[3, l, q]
            if l == 0:
                a2[:, q] = _updated(p["gues2d"].permute(0, 2, 1)[:, q], t, wbar)
    return {"anal3d": a3.permute(0, 1, 3, 2).contiguous(), "anal2d": a2.permute(0, 2, 1).contiguous(), "infl3d": i3,
            "infl2d": i3[:2, 0].clone()}


def _exact_sweep(case, seed):
    n, ne = case["nlon"] * case["nlat"] * case["nlev"], case["ne"]
    if n * (_sweep_local(case) * 3.0 * ne * ne + 40.0 * ne ** 3) > 1.0e13:
        return None
    p = _sweep_inputs(case, seed)
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=_dev())
    so, sov, dx = p["params"]["sigma_obs"], p["params"]["sigma_obsv"], p["params"]["dx"]
    ri, rj = t(p["ri"]), t(p["rj"])
    olnp = t(np.log(np.where(p["cls"] == 1, p["dat"], p["lev"])))
    einv, dep, hd = t(1.0 / p["err"] ** 2), t(p["dep"]), p["hdxf"].double()
    nlon, nlat, nlev = case["nlon"], case["nlat"], case["nlev"]
    lev = np.log(S.regional_levels(nlev))
    reach = math.sqrt(CUT2) * so / dx + 1.0e-6
    nij = nlon * nlat
    xb = p["xb"]
    xa, infl = torch.empty(xb.shape, dtype=torch.float64, device=_dev()), torch.empty_like(p["infl"])
    nobsl = torch.zeros(n, dtype=torch.int32, device=_dev())
    bs = 8
    for j0 in range(0, nlat, bs):
        for i0 in range(0, nlon, bs):
            near = ((ri > i0 + 1 - reach) & (ri < i0 + bs + reach) & (rj > j0 + 1 - reach)
                    & (rj < j0 + bs + reach)).nonzero()[:, 0]
            jj = torch.arange(j0, min(j0 + bs, nlat), device=_dev())
            ii = torch.arange(i0, min(i0 + bs, nlon), device=_dev())
            col = (jj[:, None] * nlon + ii).flatten()
            h2 = ((((col % nlon) + 1.0)[:, None] - ri[near]) * dx) ** 2 + (((col // nlon) + 1.0)[:, None] - rj[near]) \
                .mul(dx) ** 2
            h2 = h2 / so ** 2
            rows, d = hd[near], dep[near]
            yy = (rows[:, :, None] * rows[:, None, :]).flatten(1)
            for l0 in range(0, nlev, 10):
                ls = range(l0, min(l0 + 10, nlev))
                pts = torch.cat([col + l * nij for l in ls])
                nd = torch.cat([h2 + ((olnp[near] - lev[l]) / sov)[None] ** 2 for l in ls])
                inside = nd <= CUT2
                rloc = torch.exp(-0.5 * nd) * inside
                w = rloc * einv[near]
                gram = (w @ yy).reshape(-1, ne, ne)
                tr, wbar, new = _analysis(ne, gram, (w * d) @ rows, w @ d ** 2, rloc.sum(1), inside.any(1),
                                          p["infl"][pts])
                infl[pts] = new
                nobsl[pts] = inside.sum(1).int()
                xa[:, pts] = _updated(xb[:, pts].double(), tr, wbar)
    return {"xa": xa, "infl": infl, "nobsl": nobsl}


def _exact_lists(ne, p, rows_of, dep_of, weight, xb):
    """Points with packed or indexed local rows, one batch of padded lists at a time."""
    offs = p["offs"]
    n = offs.numel() - 1
    trans = torch.empty((n, ne, ne), dtype=torch.float64, device=_dev())
    transm = torch.empty((n, ne), dtype=torch.float64, device=_dev())
    infl = torch.empty_like(p["infl"])
    cnt = offs[1:] - offs[:-1]
    step = max(1, int(2.0e8 // (max(int(cnt.max()), ne, 1) * ne)))
    for q in torch.arange(n, device=_dev()).split(step):
        lm = max(int(cnt[q].max()), 1)
        within = torch.arange(lm, device=_dev())
        has = within[None] < cnt[q][:, None]
        at = (offs[q][:, None] + within).clamp(max=max(int(offs[-1]) - 1, 0))
        rows, d = rows_of(at) * has[..., None], dep_of(at)
        w, rl = weight[at] * has, p["rl"].double()[at] * has
        wr = rows * w[..., None]
        gram = torch.bmm(wr.transpose(1, 2), rows)
        b = torch.bmm(wr.transpose(1, 2), d[..., None])[..., 0]
        t, wbar, new = _analysis(ne, gram, b, (w * d * d).sum(1), rl.sum(1), cnt[q] > 0, p["infl"][q])
        trans[q], transm[q], infl[q] = t.transpose(1, 2), wbar, new
    return trans, transm, infl, _updated(xb, trans.transpose(1, 2), transm)


def _exact_core(case, seed):
    p = _core_inputs(case, seed)
    rows, dep = p["rows"].double(), p["dep"].double()
    tr, tm, infl, xa = _exact_lists(case["ne"], p, lambda a: rows[a], lambda a: dep[a], 1.0 / p["rd"].double(),
                                    p["xb"].double())
    return {"trans": tr, "transm": tm, "infl": infl, "status": None, "xa": xa}


def _exact_largek(case, seed):
    p = _largek_inputs(case, seed)
    idx = p["idx"].long()
    wt = p["rl"].double() / p["rd"].double()
    bf = case["storage"] == "bf16"
    mean, pert = p["mean"].double(), p["pert"].double()
    xb = pert if bf else (p["mean"][..., None] + p["pert"]).double()
    tr, tm, infl, xa = _exact_lists(case["ne"], p, lambda a: p["ens"][idx[a]].double(),
                                    lambda a: p["dep"][idx[a]].double(), wt, xb)
    out = {"trans": tr, "transm": tm, "infl": infl, "status": None}
    if not bf:
        return {**out, "xa": xa}
    m = pert.mean(-1, keepdim=True)
    x = pert - m
    amean = mean + m[..., 0] + torch.einsum("vpk,pk->vp", x, tm)
    return {**out, "mean": amean, "pert": torch.einsum("vpk,pmk->vpm", x, tr)}


def _exact_relax(case, seed):
    p = _relax_inputs(case, seed)
    n, ne, nv, mode = case["npts"], case["ne"], case["nv"], case["mode"]
    beta = torch.ones((nv, n), dtype=torch.float64, device=_dev())
    d = torch.minimum(torch.minimum(p["ri"] - 2, 203 - p["ri"]) * 3e3,
                      torch.minimum(p["rj"] - 2, 253 - p["rj"]) * 3e3) / 30e3
    beta = beta * torch.where(d < 1.0, d.clamp(min=0.0), torch.ones_like(d))
    if nv > 1:
        beta[1] = torch.where(p["rlev"] < 3e4, torch.zeros_like(d), beta[1])
    m = p["xb"].mean(-1, keepdim=True)
    x = p["xb"] - m
    w = p["w"]  # symmetric by construction, so its two orders are one
    al = 0.0 if mode == K.RELAX_NONE else 0.9
    fac = torch.ones((nv, n), dtype=torch.float64, device=_dev())
    if mode == K.RELAX_RTPS:
        var_a = torch.einsum("vpk,pkm,vpm->vp", x, p["pao"], x)
        var_g = (x * x).sum(-1)
        fac = torch.where(beta != 0.0, al * torch.sqrt(var_g / (var_a * (ne - 1))) - al + 1.0, fac)
    xw = torch.einsum("vpk,pkm->vpm", x, w)
    if mode == K.RELAX_RTPP:
        xw = (1.0 - al) * xw + al * x
    xw = xw * fac[..., None] + torch.einsum("vpk,pk->vp", x, p["tm"])[..., None]
    xa = m + beta[..., None] * xw + (1.0 - beta)[..., None] * x
    q = xa[0]
    qm = q.mean(-1, keepdim=True)
    sp = (q - qm).square().sum(-1, keepdim=True).div(ne - 1).sqrt() / qm
    xa[0] = torch.where(sp > 0.15, qm + (q - qm) * 0.15 / sp, q)
    return {"beta": beta, "xa": xa, "infl": fac} if mode == K.RELAX_RTPS else {"beta": beta, "xa": xa}


def _exact_obs_space(case, seed):
    p = _obs_space_inputs(case, seed)
    ne, nobs = case["ne"], case["nobs"]
    inc = 0.5 * torch.einsum("pk,pmk->pm", p["hdxf"], p["trans"]) + 0.5 * p["hdxf"]
    mode = p["mode"][:, None]
    anal = p["ybar"][:, None] + torch.where(mode == 1, p["hdxf"], inc)
    mean = torch.where(mode == 1, p["ybar"][:, None], anal.mean(1, keepdim=True))
    sp = (anal - mean).square().sum(1, keepdim=True).div(ne - 1).sqrt() / mean
    anal = torch.where((mode == 2) & (sp > 0.1), mean + (anal - mean) * 0.1 / sp, anal)
    cnt = p["offs"][1:] - p["offs"][:-1]
    point = torch.repeat_interleave(torch.arange(case["npts"], device=_dev()), cnt)
    idx = p["idx"].long()
    nterm = max(p["term"]) + 1
    djdy = torch.zeros((nobs, nterm), dtype=torch.float64, device=_dev())
    for t in range(nterm):
        w1 = sum(p["fcst"][v] * p["fcer"][v][:, None] for v in range(case["nv"]) if p["term"][v] == t)
        for c in torch.arange(idx.numel(), device=_dev()).split(500_000):
            val = (p["hdxa"][idx[c]] * w1[point[c]]).sum(1) * p["rl"][c] / p["rd"][c]
            djdy[:, t].index_add_(0, idx[c], val)
    return {"anal": anal, "mean": mean[:, 0], "djdy": djdy, "sense": djdy * p["obsdep"][:, None]}


def exact(case, seed):
    return {"ring": _exact_ring, "globe": _exact_globe, "sweep": _exact_sweep, "core": _exact_core,
            "largek": _exact_largek, "relax": _exact_relax, "obs_space": _exact_obs_space}[case["kind"]](case, seed)
