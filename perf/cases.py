"""Workloads of the LETKF library, timed through its public entry points.

A case names what a user's program asks for: one column's letkf_core, a batch of
them, a whole analysis of a globe (host arrays or device arrays, plain FP64 or
mixed precision, per column or per cube), the run_da_parallel wrapper, and the
coupler step before it.  `prepare` builds the inputs and the handle such a
program holds, `run` makes one call, `exact` restates the result in plain 64-bit
torch / numpy, and `draw` gives further cases of the same ranges.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dida-thhpca_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import letkf_gb300 as lg  # noqa: E402
import synth  # noqa: E402

FP64, MIXED, TF32 = lg.LG_PREC_FP64, lg.LG_PREC_MIXED, lg.LG_PREC_MIXED_TF32
_EARTH = 6371.393


# ------------------------------------------------------------------- the cases
def _globe(name, kind, lon, lat, nz, ens, n_obs, dist, vert, prec, **more):
    c = {"name": name, "kind": kind, "lon": lon, "lat": lat, "nz": nz, "ens": ens, "n_obs": n_obs,
         "dist": dist, "vert": vert, "prec": prec, "rho": 1.05, "nx": 8, "ny": 8, "max_obs": 10000,
         "clustered": 0.0, "cube_n": 1, "cube_nz": 1, "gc": 1}
    c.update(more)
    return c


def listed():
    return [
        # one grid column through the host-array letkf_core: a linked Fortran driver that keeps
        # its own column loop calls this once per column and level
        {"name": "core_one_column", "kind": "core_host", "ens": 40, "p": 180, "rho": 1.05},
        # a driver with its own selection: the columns of one latitude band and level in one batch
        {"name": "core_batch_40", "kind": "core", "ens": 40, "nbatch": 2304, "p": 300, "prec": FP64,
         "rho": 1.05},
        # the same with 64 members, long lists and tensor-core contractions
        {"name": "core_batch_64_mixed", "kind": "core", "ens": 64, "nbatch": 1440, "p": 900,
         "prec": MIXED, "rho": 1.05},
        # the 5-degree single-level set-up (72 x 36, 16 members, 2000 observations): one cycle --
        # new observations, then letkf_run on host arrays; the smallest whole analysis
        _globe("cycle_one_level_16", "cycle", 72, 36, 1, 16, 2000, 1000.0, -1.0, FP64, nx=4, ny=4,
               rho=1.1),
        # a coarse 3-D cycle on host arrays (72 x 36 x 32, 40 members, 4000 observations)
        _globe("cycle_coarse_40", "cycle", 72, 36, 32, 40, 4000, 1000.0, 0.2, FP64, nx=4, ny=4),
        # the plain-FP64 drop-in at 1.5 degrees: 40 members, 10^5 observations, resident arrays
        _globe("globe_40", "resident", 240, 120, 32, 40, 100_000, 800.0, 0.2, FP64),
        # plain FP64 at 64 members where observations are dense (lists of some thousands)
        _globe("globe_dense_64", "resident", 90, 45, 32, 64, 250_000, 800.0, 0.2, FP64, max_obs=0),
        # mixed precision at 64 members: the main configuration on a 2-degree grid
        _globe("globe_64_mixed", "resident", 180, 90, 32, 64, 250_000, 800.0, 0.2, MIXED, max_obs=0),
        # mixed precision at 128 members with half of the observations in clusters
        _globe("globe_128_mixed", "resident", 48, 24, 32, 128, 60_000, 500.0, 0.2, MIXED, max_obs=0,
               rho=1.03, nx=4, ny=4, clustered=0.5),
        # cube analyses (da_block_interval 2, da_vertical_interval 2), plain FP64
        _globe("cubes_40", "resident", 120, 60, 32, 40, 25_000, 800.0, 0.2, FP64, cube_n=2,
               cube_nz=2),
        # run_da_parallel: full members in host memory in, blended members and spreads out
        _globe("da_parallel_20", "da_parallel", 60, 30, 32, 20, 6000, 1000.0, 0.2, FP64, nx=4, ny=4),
        # the coupler step: GMCORE's C grid to the background layout, 64 members at 2 degrees
        {"name": "coupler_64", "kind": "coupler", "lon": 180, "lat": 90, "nz": 32, "ens": 64},
    ]


def _between(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["core_host", "core", "core", "cycle", "resident", "resident", "resident",
                       "resident", "cubes", "da_parallel", "coupler"])
    if kind == "core_host":
        return {"kind": kind, "ens": _between(rng, 8, 128), "p": _between(rng, 1, 3000), "rho": 1.05}
    if kind == "core":
        ens = _between(rng, 8, 128)
        most = min(4096, int(3.8e8 / ens ** 3))
        prec = rng.choice([FP64, FP64, MIXED, TF32])
        if prec == TF32 and ens > 64:
            prec = MIXED
        return {"kind": kind, "ens": ens, "nbatch": _between(rng, min(64, most), most),
                "p": _between(rng, 20, 1500), "prec": prec, "rho": round(rng.uniform(1.0, 1.2), 3)}
    if kind == "coupler":
        return {"kind": kind, "lon": rng.randrange(40, 181), "lat": rng.randrange(20, 91),
                "nz": rng.choice([8, 20, 32]), "ens": _between(rng, 5, 64)}
    lon = _between(rng, 48, 180)
    c = _globe("", kind, lon, max(24, lon // 2 + rng.randrange(-3, 4)), rng.choice([1, 8, 20, 32, 32]),
               _between(rng, 8, 100), 0, float(rng.randrange(400, 1201, 50)),
               round(rng.uniform(0.1, 0.4), 2), rng.choice([FP64, FP64, MIXED, MIXED, TF32]),
               rho=round(rng.uniform(1.0, 1.2), 3), clustered=rng.choice([0.0, 0.0, 0.5]))
    c["n_obs"] = _between(rng, 1000, 120_000)
    del c["name"]
    if c["prec"] == TF32 and c["ens"] > 64:
        c["prec"] = MIXED
    if rng.random() < 0.15:
        c["gc"] = 0  # box localisation
    if c["nz"] == 1:
        c["vert"] = -1.0
    if kind == "cubes":
        c.update(kind="resident", cube_n=rng.choice([2, 3]), cube_nz=rng.choice([1, 2, 3]))
        c["prec"] = min(c["prec"], MIXED)
    if kind in ("cycle", "da_parallel"):
        c.update(lon=min(c["lon"], 72), lat=min(c["lat"], 36), ens=min(c["ens"], 40),
                 n_obs=min(c["n_obs"], 10_000), prec=FP64, nx=4, ny=4)
    while _seconds(c) > 0.8:  # no more than the largest listed case costs
        if c["n_obs"] > 4000:
            c["n_obs"] = int(c["n_obs"] * 0.7)
        else:
            c["lon"], c["lat"] = int(c["lon"] * 0.8), max(16, int(c["lat"] * 0.8))
    return c


def _config(c):
    names = ("x",) if c["nz"] == 1 else ("ps", "u", "v", "pt")
    sig = {"x": 0.5, "ps": 100.0, "u": 1.0, "v": 1.0, "pt": 0.5}
    return lg.Config("case", c["ens"], c["lat"], c["lon"], c["nz"], names, c["dist"], c["vert"],
                     c["rho"], c["n_obs"], c["nx"], c["ny"], max_obs=c["max_obs"],
                     gc_filter=c["gc"], gc_filter_vertical=c["gc"], precision=c["prec"],
                     obs_sigma={v: sig[v] for v in names}, sh_degree=10,
                     vcoord=lg.LG_VCOORD_SIGMA if c["nz"] == 1 else lg.LG_VCOORD_HYBRID,
                     clustered_frac=c["clustered"], cube_n=c["cube_n"], cube_nz=c["cube_nz"])


# ------------------------------------------------------------------ the work
def _solves(c):
    """(solves, list entries with a weight per solve) of one analysis, on average."""
    p = c["n_obs"] * (1.0 - math.cos(min(math.pi, 2.0 * c["dist"] / _EARTH))) / 2.0
    cols = c["lon"] * c["lat"] / c["cube_n"] ** 2
    if c["max_obs"]:
        p = min(p, c["max_obs"])
    if c["vert"] <= 0:
        return cols, p
    a, b, p0, ptop = lg.vertical_coord(_config(c))
    half = a * (p0 - ptop) + b * (1e5 - ptop) + ptop
    z = np.log(0.5 * (half[1:] + half[:-1]))
    share = float((np.abs(z[:, None] - z[None, :]) <= 2.0 * c["vert"]).mean())
    return cols * c["nz"] / c["cube_nz"], p * share


def _rows(c):
    return 1 if c["nz"] == 1 else 1 + 3 * c["nz"]


def _seconds(c):
    """A rough time of an analysis, to bound what draw() asks for."""
    s, p = _solves(c)
    k = c["ens"]
    gram = s * p * k * k * (1.6e-12 if c["prec"] == FP64 else 1e-13)
    return gram + s * k ** 3 * (1.2e-11 if c["cube_n"] > 1 and c["prec"] == FP64 else 4e-12)


def work(c):
    k = c["ens"]
    if c["kind"] == "coupler":
        pts = c["lon"] * c["lat"] * k
        out = (c["lon"] + 2) * c["lat"] * k * (1 + 3 * c["nz"])
        return {"bytes": 8.0 * (pts * (1 + 3 * c["nz"]) + c["lon"] * k * c["nz"] + out),
                "flops": 4.0 * pts * c["nz"]}
    if c["kind"] in ("core", "core_host"):
        n = c.get("nbatch", 1)
        # Gram (one triangle) and projection, eigen-decomposition, trans and overline_w
        flops = n * (c["p"] * (k * (k + 1) + 2 * k) + 9.0 * k ** 3 + 2.0 * k ** 3)
        return {"bytes": n * (c["p"] * (8.0 * k + 20) + 8.0 * (k * k + k)), "flops": flops}
    s, p = _solves(c)
    cols, rows = c["lon"] * c["lat"], _rows(c)
    # Gram and projection, reduction to tridiagonal form, its square root applied to the rows
    flops = s * (p * (k * (k + 1) + 2 * k) + 4.0 / 3 * k ** 3) + cols * rows * 8.0 * k * k
    cells = (c["lon"] + 2) * (c["lat"] + 2) * rows
    return {"bytes": 8.0 * (2 * cells * (k + 1)) + 44.0 * c["n_obs"], "flops": flops}


# ------------------------------------------------------------------ the inputs
def _core_inputs(c, seed):
    """Ensemble perturbations in observation space, errors, departures and weights of each
    batch member, with list lengths spread around p (some of them empty)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, n = c["ens"], c.get("nbatch", 1)
    if n > 1:
        cnt = (c["p"] * 2.0 * torch.rand(n, generator=g, device="cuda")).int()
        cnt[:: 97] = 0
    else:
        cnt = torch.full((1,), c["p"], dtype=torch.int32, device="cuda")
    off = torch.cumsum(cnt.long(), 0) - cnt.long()
    tot = max(1, int(cnt.sum()))
    f64 = dict(dtype=torch.float64, device="cuda", generator=g)
    hx = torch.randn((tot, k), **f64)
    hx -= hx.mean(dim=1, keepdim=True)
    sd = 0.5 + 1.5 * torch.rand(tot, **f64)
    rd = (1.0 / (sd * sd)).float()
    dep = torch.randn(tot, **f64) * 1.5
    ri = 2.0 * torch.sqrt(torch.rand(tot, **f64))  # uniform over the localisation disc
    return cnt, off, hx, rd, dep, _taper(ri)


def _workload(c, seed):
    cfg = _config(c).replace(seed=seed)
    return cfg, synth.make_workload(cfg, backend="torch", device=torch.device("cuda"))


def prepare(c, seed):
    kind = c["kind"]
    if kind == "coupler":
        g = torch.Generator(device="cuda").manual_seed(seed)
        nz, nla, nlo, k = c["nz"], c["lat"], c["lon"], c["ens"]
        f64 = dict(dtype=torch.float64, device="cuda", generator=g)
        area = torch.cos(torch.linspace(-1.5, 1.5, nla, dtype=torch.float64, device="cuda"))
        sub = area[:, None] * (0.4 + 0.2 * torch.rand((nla, 2), **f64))
        return {"kind": kind, "args": [1e5 + 500 * torch.randn((nla, nlo, k), **f64),
                                       10 * torch.randn((nz, nla, nlo, k), **f64),
                                       10 * torch.randn((nz, nla + 1, nlo, k), **f64),
                                       300 + 5 * torch.randn((nz, nla, nlo, k), **f64),
                                       sub, sub.sum(dim=1)]}
    if kind in ("core", "core_host"):
        ins = _core_inputs(c, seed)
        if kind == "core_host":
            return {"kind": kind, "rho": c["rho"], "args": [t.cpu().numpy() for t in ins[2:]]}
        n, k = c["nbatch"], c["ens"]
        return {"kind": kind, "ins": ins, "k": k, "n": n, "rho": c["rho"], "prec": c["prec"],
                "lib": lg.load_library(),
                "trans": torch.empty((n, k, k), dtype=torch.float64, device="cuda"),
                "wbar": torch.empty((n, k), dtype=torch.float64, device="cuda")}
    cfg, w = _workload(c, seed)
    s = {"kind": kind, "ctx": lg.Letkf(cfg), "obs": w.obs}
    if kind == "resident":
        s["ctx"].set_obs(w.obs)
        s.update(xb=w.xb, axb=w.axb, xa=torch.zeros_like(w.xb), axa=torch.zeros_like(w.axb))
    elif kind == "cycle":
        s.update(xb=w.xb.cpu().numpy(), axb=w.axb.cpu().numpy())
        s.update(xa=np.zeros_like(s["xb"]), axa=np.zeros_like(s["axb"]))
    else:
        full = (w.xb + w.axb[..., None]).cpu().numpy()
        spread = np.zeros((cfg.num_lon, cfg.num_lat, cfg.n_rows))
        s.update(full=full, out=np.zeros_like(full), sb=spread, sa=spread.copy())
    return s


# -------------------------------------------------------------------- one pass
_GAMMA1, _GAMMA2, _POLAR = 0.3, 0.7, 85.0


def run(s):
    kind = s["kind"]
    if kind == "coupler":
        return lg.gmcore_to_da(*s["args"], halo=1)
    if kind == "core_host":
        return list(lg.letkf_core(*s["args"], s["rho"]))
    if kind == "core":
        p = [C.c_void_p(t.data_ptr()) for t in s["ins"]]
        lg.check(s["lib"].lg_core_batch(s["k"], s["n"], *p, s["rho"], s["prec"],
                                        C.c_void_p(s["trans"].data_ptr()),
                                        C.c_void_p(s["wbar"].data_ptr()),
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return [s["trans"], s["wbar"]]
    ctx = s["ctx"]
    if kind == "resident":
        ctx.letkf_run_device(0, s["xb"], s["axb"], s["xa"], s["axa"])
        return [s["xa"], s["axa"]]
    ctx.set_obs(s["obs"])
    if kind == "cycle":
        ctx.letkf_run(0, s["xb"], s["axb"], s["xa"], s["axa"])
        return [s["xa"], s["axa"]]
    ctx.run_da_parallel(0, _GAMMA1, _GAMMA2, _POLAR, s["full"], s["out"], s["sb"], s["sa"])
    return [s["out"], s["sb"], s["sa"]]


# ------------------------------------------------------- the result in 64 bits
def _taper(r):
    """Gaspari-Cohn with the single-precision literals the path defines."""
    c1, c2 = float(np.float32(1.666667)), float(np.float32(0.6666667))
    near = ((((-0.25 * r + 0.5) * r + 0.625) * r - c1) * (r * r)) + 1.0
    rs = r.clamp(min=1e-3)
    far = ((((r / 12.0 - 0.5) * r + 0.625) * r + c1) * r - 5.0) * r + 4.0 - c2 / rs
    return torch.where(r > 2.0, torch.zeros_like(r), torch.where(r > 1.0, far, near))


def _core64(gram, t, rho):
    """(W, overline_w) of [S, k, k] Gram matrices and [S, k] projections."""
    k = gram.shape[-1]
    if gram.shape[0] <= 4096:
        lam, v = np.linalg.eigh(gram.cpu().numpy())
        lam, v = torch.as_tensor(lam).cuda() + (k - 1) / rho, torch.as_tensor(v).cuda()
        w = (v * torch.sqrt((k - 1) / lam)[:, None, :]) @ v.transpose(1, 2)
        return w, (v @ ((v.transpose(1, 2) @ t[..., None]) / lam[..., None]))[..., 0]
    return _core64_many(gram, t, rho)


def _core64_many(gram, t, rho):
    """As _core64, by the coupled Newton-Schulz iteration for A^-1/2 (many small matrices)."""
    k = gram.shape[-1]
    eye = torch.eye(k, dtype=torch.float64, device="cuda")
    a = gram + (k - 1) / rho * eye
    s = a.abs().sum(dim=2).max(dim=1).values[:, None, None]
    y, z = a / s, eye.expand_as(a).clone()
    for _ in range(60):
        m = z @ y
        if float((m - eye).abs().max()) < 1e-13:
            break
        step = 1.5 * eye - 0.5 * m
        y, z = y @ step, step @ z
    z = z / torch.sqrt(s)
    return math.sqrt(k - 1) * z, (z @ (z @ t[..., None]))[..., 0]


def _exact_core(c, seed):
    cnt, off, hx, rd, dep, rloc = _core_inputs(c, seed)
    rr = torch.sqrt(rd.double() * rloc)
    h = hx * rr[:, None]
    k = c["ens"]
    gram = torch.zeros((cnt.numel(), k, k), dtype=torch.float64, device="cuda")
    t = torch.zeros((cnt.numel(), k), dtype=torch.float64, device="cuda")
    for i, (n, o) in enumerate(zip(cnt.tolist(), off.tolist())):
        a = h[o:o + n]
        gram[i] = a.T @ a
        t[i] = a.T @ (rr[o:o + n] * dep[o:o + n])
    w, wbar = _core64(gram, t, c["rho"])
    # column-major trans(i, j) = W(i, j) + overline_w(i)
    trans = (w + wbar[:, :, None]).transpose(1, 2).contiguous()
    return trans, wbar


def _blocks(cfg):
    """(first, last) latitude / longitude index (0-based, last excluded) of every block."""
    def cut(n, parts):
        sec, res = divmod(n, parts)
        ends = np.cumsum([sec + (i < res) for i in range(parts)])
        return np.concatenate([[0], ends[:-1]]), ends
    return cut(cfg.num_lat, cfg.global_nx), cut(cfg.num_lon, cfg.global_ny)


def _gc_dist(la1, lo1, la2, lo2, f=np.float64):
    pi = f(np.float32(np.arctan(np.float32(1.0)) * np.float32(4.0)))
    r = lambda x: f(x) / f(180.0) * pi  # noqa: E731
    v = np.cos(r(la1)) * np.cos(r(la2)) * np.cos(r(lo1) - r(lo2)) + np.sin(r(la1)) * np.sin(r(la2))
    return f(np.float32(6371.393)) * np.arccos(np.minimum(f(v), f(1.0)))


def _neighbours(cfg, gl, gn):
    """Neighbour blocks of every block, in the order the selection walks them."""
    (s1, e1), (s2, e2) = _blocks(cfg)
    nx, ny, far = cfg.global_nx, cfg.global_ny, cfg.local_dist

    def gap(bx, by, tx, ty):
        if bx != tx:
            p, q = (s1[bx], e1[tx]) if bx > tx else (e1[bx], s1[tx])
        else:
            p, q = (e1[bx], e1[tx]) if bx + 1 > nx // 2 else (s1[bx], s1[tx])
        if by == ty:
            return _gc_dist(gl[p], gn[s2[by]], gl[q], gn[s2[ty]], np.float32)
        n = cfg.num_lon
        return min(_gc_dist(gl[p], gn[s2[by]], gl[q], gn[e2[ty] % n], np.float32),
                   _gc_dist(gl[p], gn[e2[by] % n], gl[q], gn[s2[ty]], np.float32))

    table = {}
    for by in range(ny):
        for bx in range(nx):
            lo, hi, ref = bx, bx, gn[s2[by]]
            while lo > 0 and _gc_dist(gl[s1[bx]], ref, gl[e1[lo - 1]], ref) <= far:
                lo -= 1
            while hi < nx - 1 and _gc_dist(gl[e1[bx]], ref, gl[s1[hi + 1]], ref) <= far:
                hi += 1
            out = []
            for tx in range(lo, hi + 1):
                west = east = 0
                while west <= (ny - 1) // 2 and gap(bx, by, tx, (by - west - 1) % ny) <= far:
                    west += 1
                while east <= (ny - 1) // 2 and gap(bx, by, tx, (by + east + 1) % ny) <= far:
                    east += 1
                if west + east > ny - 1:
                    east -= 1
                out += [(tx, (by + j) % ny) for j in range(-west, east + 1)]
            table[bx, by] = out
    return table


def _half_levels(cfg, ps):
    a, b, p0, ptop = (torch.as_tensor(x, device="cuda") if isinstance(x, np.ndarray) else x
                      for x in lg.vertical_coord(cfg))
    if cfg.vcoord == lg.LG_VCOORD_SIGMA:
        half = a * (ps[..., None] - ptop) + ptop
    else:
        half = a * (p0 - ptop) + b * (ps[..., None] - ptop) + ptop
    return 0.5 * (half[..., 1:] + half[..., :-1])


def _observed(cfg, x, obs, gl, gn):
    """Members interpolated to every observation [n_obs, k] (x: full members)."""
    dev = dict(device="cuda")
    la = np.searchsorted(gl.astype(np.float64), obs.lat)
    lo = np.searchsorted(gn.astype(np.float64), obs.lon)
    dla = (gl[la] - gl[np.maximum(la - 1, 0)]).astype(np.float64)
    dlo = (gn[lo] - gn[np.maximum(lo - 1, 0)]).astype(np.float64)
    with np.errstate(divide="ignore", invalid="ignore"):
        ax = np.where(la > 0, (dla - obs.lat + gl[np.maximum(la - 1, 0)]) / dla, 0.0)
        ay = np.where(lo > 0, (dlo - obs.lon + gn[np.maximum(lo - 1, 0)]) / dlo, 0.0)
    la, lo = torch.as_tensor(la, **dev) + cfg.halo, torch.as_tensor(lo, **dev) + cfg.halo
    ax, ay = torch.as_tensor(ax, **dev)[:, None], torch.as_tensor(ay, **dev)[:, None]
    m = torch.arange(cfg.ens, **dev)[None]

    def at(row):
        cell = lambda i, j: x[j[:, None], i[:, None], row, m]  # noqa: E731
        west = cell(la - 1, lo - 1) * ax + cell(la, lo - 1) * (1 - ax)
        east = cell(la - 1, lo) * ax + cell(la, lo) * (1 - ax)
        return west * ay + east * (1 - ay)

    mid = _half_levels(cfg, at(torch.zeros_like(la)[:, None]))  # [n_obs, k, nz]
    ph = torch.as_tensor(obs.ph, **dev)
    pos = (mid < ph[:, None, None]).sum(dim=2)
    start = torch.as_tensor(np.concatenate([[0], np.cumsum(cfg.var_lev)[:-1]]), **dev)
    levs = torch.as_tensor(np.asarray(cfg.var_lev), **dev)
    var = torch.as_tensor(np.asarray([t[2][0] for t in obs.types])[obs.type], **dev)
    s, lv = start[var][:, None], levs[var][:, None]
    inner = (pos >= 1) & (pos < cfg.nz) & (lv > 1)
    up = torch.where(lv > 1, s + (pos - 1).clamp(0, cfg.nz - 1), s)
    dn = torch.where(inner, up + 1, up)
    hi = torch.log(mid.gather(2, pos.clamp(max=cfg.nz - 1)[..., None])[..., 0])
    lw = torch.log(mid.gather(2, (pos - 1).clamp(min=0)[..., None])[..., 0])
    t3 = torch.where(inner, (hi - torch.log(ph)[:, None]) / torch.where(inner, hi - lw, torch.ones_like(hi)),
                     torch.ones_like(hi))
    return at(up) * t3 + at(dn) * (1 - t3)


def _exact_analysis(cfg, xb, axb, obs):
    """(xa, axa) of the whole globe, per column or per cube, halo points zero."""
    gl, gn = lg.model_grid(cfg)
    h, k, nz = cfg.halo, cfg.ens, cfg.nz
    y = _observed(cfg, xb + axb[..., None], obs, gl, gn)
    dep = torch.as_tensor(obs.yo, device="cuda") - y.mean(dim=1)
    y = y - y.mean(dim=1, keepdim=True)
    rd = torch.as_tensor(obs.rinv, device="cuda").float().double()
    lnp = torch.log(torch.as_tensor(obs.ph, device="cuda"))
    (s1, e1), (s2, e2) = _blocks(cfg)
    box = lambda v: float("%.5f" % v)  # noqa: E731
    held = {}
    for by in range(cfg.global_ny):
        for bx in range(cfg.global_nx):
            m = ((obs.lon >= box(gn[s2[by]])) & (obs.lon <= box(gn[e2[by]])) &
                 (obs.lat >= box(gl[s1[bx]])) & (obs.lat <= box(gl[e1[bx]])))
            o = np.nonzero(m)[0]
            held[bx, by] = o[np.argsort(obs.type[o], kind="stable")]
    vertical = cfg.vert_dist > 0
    step = cfg.cube_nz if vertical else 1
    groups = [(a, min(a + step, nz)) for a in range(0, nz, step)] if vertical else [(0, nz)]
    taper = _taper if cfg.gc_filter else (lambda r: (r <= 2.0).double())
    taperz = _taper if cfg.gc_filter_vertical else (lambda r: (r <= 2.0).double())
    rows = {}  # rows analysed by each level group
    for i, (a, b) in enumerate(groups):
        rows[i] = []
        for st, lv in zip(np.concatenate([[0], np.cumsum(cfg.var_lev)[:-1]]), cfg.var_lev):
            if lv == 1:
                rows[i] += [int(st)] if i == len(groups) - 1 else []
            else:
                rows[i] += [int(st) + r for r in range(a, b)]
    xa, axa = torch.zeros_like(xb), torch.zeros_like(axb)
    for (bx, by), near in _neighbours(cfg, gl, gn).items():
        cand = np.concatenate([held[b] for b in near])
        ci = torch.as_tensor(cand, device="cuda")
        cubes = [(j, min(j + cfg.cube_n, e1[bx]), i, min(i + cfg.cube_n, e2[by]))
                 for i in range(s2[by], e2[by], cfg.cube_n) for j in range(s1[bx], e1[bx], cfg.cube_n)]
        # the centre grid point, from block-local 1-based indices
        mid = lambda s, e, o: o + ((s - o + 1) + (e - o)) // 2 - 1  # noqa: E731
        cla = np.array([mid(q[0], q[1], s1[bx]) for q in cubes])
        clo = np.array([mid(q[2], q[3], s2[by]) for q in cubes])
        cut = lambda v: torch.as_tensor(np.asarray(v, np.float64), device="cuda")  # noqa: E731
        pi = float(np.float32(np.arctan(np.float32(1.0)) * np.float32(4.0)))
        la1, lo1 = cut(obs.lat[cand]) / 180 * pi, cut(obs.lon[cand]) / 180 * pi
        la2, lo2 = cut(gl[cla])[:, None] / 180 * pi, cut(gn[clo])[:, None] / 180 * pi
        v = torch.cos(la1) * torch.cos(la2) * torch.cos(lo1 - lo2) + torch.sin(la1) * torch.sin(la2)
        ri = float(np.float32(6371.393)) * torch.acos(v.clamp(max=1.0)) / cfg.local_dist
        wgt = taper(ri) * (cut(np.abs(obs.lat[cand])) <= cfg.obs_polar)
        if cfg.max_obs:
            wgt = wgt * (torch.cumsum((wgt > 0).int(), dim=1) <= cfg.max_obs)
        ps = axb[torch.as_tensor(clo, device="cuda") + h, torch.as_tensor(cla, device="cuda") + h, 0]
        lnl = torch.log(_half_levels(cfg, ps))
        for i, (a, b) in enumerate(groups):
            use = wgt
            if vertical:
                centre = (a + 1 + b) // 2 - 1
                use = wgt * taperz((lnl[:, centre, None] - lnp[ci][None]).abs() / cfg.vert_dist)
            keep = (use > 0).any(dim=0)
            rr = torch.sqrt(rd[ci[keep]][None] * use[:, keep])
            part = max(1, int(4e8 / max(1, rr.shape[1] * k)))
            gram = torch.empty((len(cubes), k, k), dtype=torch.float64, device="cuda")
            t = torch.empty((len(cubes), k), dtype=torch.float64, device="cuda")
            for q in range(0, len(cubes), part):
                f = rr[q:q + part, :, None] * y[ci[keep]][None]
                gram[q:q + part] = f.transpose(1, 2) @ f
                t[q:q + part] = (f * (rr[q:q + part] * dep[ci[keep]][None])[..., None]).sum(dim=1)
            w, wbar = _core64_many(gram, t, cfg.inflation)
            for di in range(cfg.cube_n):
                for dj in range(cfg.cube_n):
                    sel = [n for n, q in enumerate(cubes) if q[0] + dj < q[1] and q[2] + di < q[3]]
                    if not sel:
                        continue
                    jo = torch.as_tensor([cubes[n][2] + di + h for n in sel], device="cuda")[:, None]
                    ja = torch.as_tensor([cubes[n][0] + dj + h for n in sel], device="cuda")[:, None]
                    r = torch.as_tensor(rows[i], device="cuda")[None]
                    x = xb[jo, ja, r]
                    n = torch.as_tensor(sel, device="cuda")
                    new = x @ w[n] + (x @ wbar[n][..., None]) + axb[jo, ja, r][..., None]
                    mean = new.mean(dim=2)
                    axa[jo, ja, r] = mean
                    xa[jo, ja, r] = new - mean[..., None]
    return xa, axa


def exact(c, seed):
    kind = c["kind"]
    if kind == "coupler":
        ps, u, v, pt, sub, area = prepare(c, seed)["args"]
        nz, nla, nlo, k = u.shape
        out = torch.zeros((nlo + 2, nla + 2, 1 + 3 * nz, k), dtype=torch.float64, device="cuda")
        uc = 0.5 * (u + torch.roll(u, 1, dims=2))
        f = 2.0 * sub / area[:, None]
        vc = v[:, :-1] * f[None, :, 0, None, None] + v[:, 1:] * f[None, :, 1, None, None]
        new = torch.cat([ps[None], uc, vc, pt]).permute(2, 1, 0, 3)
        out[1:-1, 1:-1] = new
        out[0, 1:-1], out[-1, 1:-1] = new[-1], new[0]
        return out
    if kind == "core_host":
        trans, wbar = _exact_core(c, seed)
        return [trans[0], wbar[0]]
    if kind == "core":
        return list(_exact_core(c, seed))
    s, p = _solves(c)
    # the dense products below weigh every candidate of the neighbour blocks
    if s * c["n_obs"] * c["ens"] ** 2 * 0.5 + s * c["ens"] ** 3 * 120 > 8e12:
        return None
    cfg, w = _workload(c, seed)
    if kind != "da_parallel":
        return list(_exact_analysis(cfg, w.xb, w.axb, w.obs))
    full = w.xb + w.axb[..., None]
    axb = full.mean(dim=3)
    xb = full - axb[..., None]
    xa, axa = _exact_analysis(cfg, xb, axb, w.obs)
    lat, _ = lg.model_grid(cfg)
    inner = torch.as_tensor(np.abs(lat[:-1]) <= _POLAR, device="cuda")[None, :, None, None]
    i = slice(1, -1)
    old = (axb[..., None] + xb)[i, i]
    new = torch.where(inner, _GAMMA1 * old + _GAMMA2 * (axa[..., None] + xa)[i, i], old)
    out = torch.zeros_like(full)
    out[i, i] = new
    sb = torch.sqrt((xb[i, i] ** 2).sum(dim=3) / cfg.ens)
    sa = torch.sqrt(((new - axa[i, i, :, None]) ** 2).sum(dim=3) / cfg.ens)
    return [out, sb, torch.where(inner[..., 0], sa, sb)]
