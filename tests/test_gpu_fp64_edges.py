"""Edges of the plain-FP64 path: spectra and magnitudes outside its kernels' ranges,
zero rows, boundaries of the localisation, and what its entry points keep and report.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_ft import _check
from test_gpu_gram64 import LG_ERR_EIG, _batch, _case, _reference
from test_gpu_parity import RTOL_ANALYSIS, _rel_err, _run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [7, 40, 64])
def test_core_spectra_beyond_the_node_table(k):
    """Full-rank Gram matrices up to 2^400 times (k - 1) / rho: beyond 2^40 the
    eigenvalue route answers.  f(T) in units of 2^-62 of sqrt(rho) leaves W some 2^-40 of
    itself at that line, 1e-12, beside k 2^-53 of the reference; 1e-9 has room for both."""
    rng = np.random.default_rng(40 + k)
    cases = []
    for scale in (2.0 ** 14, 2.0 ** 20, 2.0 ** 45, 2.0 ** 120, 2.0 ** 200):
        hx = rng.standard_normal((6 * k, k))  # of full rank: the members' mean stays
        cases.append((hx * scale, np.ones(6 * k, np.float32), rng.standard_normal(6 * k),
                      rng.uniform(0.5, 1.0, 6 * k)))
    cases.append(_case(rng, k, 300))
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    _check(cases.pop(), 1.05, tr[-1], wb[-1])
    for c, t, w in zip(cases, tr, wb):
        lam = np.linalg.eigvalsh((c[0] * c[3][:, None]).T @ c[0])
        size = np.sqrt((k - 1) / max(lam.min(), (k - 1) / 1.05))  # of W, for this full-rank C
        t0, w0 = _reference(*c, 1.05)
        assert np.abs(w - w0).max() <= 1e-9 * max(np.abs(w0).max(), 1e-300)
        assert np.abs((t - w) - (t0.T - w0[:, None]).T).max() <= 1e-9 * size


@pytest.mark.parametrize("name,ens,more", [
    ("tiny3d", 16, {}), ("tiny3d", 64, {}), ("tiny2d", 8, {}),
    ("tiny3d", 16, {"cube_n": 2, "cube_nz": 2}), ("tiny3d", 16, {"cube_n": 3, "overlap": 1})])
def test_analysis_spectra_beyond_the_node_table(name, ens, more, monkeypatch):
    """Observation errors of 1e-18: every column's Gram matrix is far beyond the table, so
    the analysis is the accumulating eigenvalue solver's bit for bit -- the solver that a
    lowered sweep limit with a rotation log of one octet gives (cubes: the limit alone)."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset(name).replace(ens=ens, local_dist=9000.0, vert_dist=3.0 if "3d" in name else -1.0,
                                  **more)
    w = synth.make_workload(cfg)
    w.obs.rinv[:] = 1e36
    out = []
    for old in (False, True):
        if old:
            monkeypatch.setenv("LETKF_GB300_QL_ITERS", "59")
            monkeypatch.setenv("LETKF_GB300_ROT_CAP", "8")
        ctx = lg.Letkf(cfg)
        ctx.set_obs(w.obs)
        xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
        st = 0
        try:
            ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        except RuntimeError as e:
            st = str(e)
        out.append((xa, axa, st, ctx.stats()["n_eig_fail"]))
        ctx.letkf_final()
    assert out[0][2:] == out[1][2:]
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)
    assert np.array_equal(out[0][1], out[1][1], equal_nan=True)


def test_spectra_beyond_the_node_table_at_every_core_entry():
    """lg_letkf_core and lg_core_batch_noalloc answer such a solve as lg_core_batch does, a
    usual one beside it too."""
    import torch
    import letkf_gb300 as lg
    L = lg.load_library()
    rng = np.random.default_rng(3)
    k, p = 24, 150
    cases = [_case(rng, k, p), (rng.standard_normal((p, k)) * 2.0 ** 45, np.ones(p, np.float32),
                                rng.standard_normal(p), np.ones(p))]
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    for c, t, w in zip(cases, tr, wb):
        t1, w1 = lg.letkf_core(*c, 1.05)
        assert np.array_equal(t1, t) and np.array_equal(w1, w)
    dev = [torch.from_numpy(np.array([p, p], np.int32)).cuda(), torch.tensor([0, p]).cuda()]
    dev += [torch.from_numpy(np.concatenate([c[i] for c in cases])).cuda() for i in range(4)]
    outs = [torch.zeros(s, dtype=torch.float64, device="cuda") for s in ((2, k, k), (2, k))]
    P = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    L.lg_core_batch_noalloc.argtypes = L.lg_core_batch.argtypes
    assert L.lg_core_batch_noalloc(k, 2, *[P(d) for d in dev], 1.05, 0, P(outs[0]), P(outs[1]),
                                   None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(outs[0].cpu().numpy(), tr) and np.array_equal(outs[1].cpu().numpy(), wb)


@pytest.mark.parametrize("name,ens", [("tiny2d", 8), ("tiny3d", 16), ("tiny3d", 64)])
def test_a_variable_that_is_zero_stays_zero(name, ens):
    """Members without spread around a zero mean: every term of such a row's analysis is
    zero, so xa and axa are exactly zero."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset(name).replace(ens=ens)
    w = synth.make_workload(cfg)
    rows = slice(0, 1) if cfg.nz == 1 else slice(1 + cfg.nz, 1 + 2 * cfg.nz)  # x, or v
    w.xb[:, :, rows] = 0.0
    w.axb[:, :, rows] = 0.0
    xa, axa = np.full_like(w.xb, np.nan), np.full_like(w.axb, np.nan)
    ctx = lg.Letkf(cfg)
    ctx.set_obs(w.obs)
    ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    ctx.letkf_final()
    i = slice(cfg.halo, -cfg.halo)
    assert not axa[i, i, rows].any()
    assert not xa[i, i, rows].any()


def test_box_localisation_at_exactly_two_scales():
    """An observation whose |ln p - ln p_e| / vert_dist is exactly 2 belongs to the box
    (weight 1), and with the next smaller vert_dist it does not.  Twelve levels, each with a
    vert_dist of half its own distance; with that next one the product with the rounded
    reciprocal would still be 2 for some."""
    import torch
    import letkf_gb300 as lg
    import synth
    base = lg.preset("tiny3d").replace(nz=12, gc_filter=0, gc_filter_vertical=0, n_obs=40)
    w = synth.make_workload(base)
    w.axb[:, :, 0] = 1e5
    w.obs.type[:] = 0  # ps: no level search in H(x)
    w.obs.ph[:] = 2e4
    w.obs.yo[:] = 1e5 + 500.0
    a, b, p0, ptop = lg.vertical_coord(base)
    lev = a * (p0 - ptop) + b * (1e5 - ptop) + ptop
    dz = (torch.log(torch.from_numpy(0.5 * (lev[:-1] + lev[1:])).cuda())
          - torch.log(torch.tensor(2e4, dtype=torch.float64, device="cuda"))).abs().cpu().numpy()
    within = 0
    for kk in range(base.nz):
        cfg = base.replace(vert_dist=float(dz[kk] / 2.0))
        less = np.nextafter(cfg.vert_dist, 0.0)
        assert dz[kk] / cfg.vert_dist == 2.0 < dz[kk] / less
        within += dz[kk] * (1.0 / less) <= 2.0
        out = []
        for vd in (cfg.vert_dist, less):
            ctx = lg.Letkf(cfg.replace(vert_dist=float(vd)))
            ctx.set_obs(w.obs)
            xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
            ctx.letkf_run(0, w.xb, w.axb, xa, axa)
            ctx.letkf_final()
            out.append(axa[1:-1, 1:-1, 1 + kk] - w.axb[1:-1, 1:-1, 1 + kk])
        assert np.abs(out[0]).max() > 1e-6    # u at this level is analysed from the observations
        assert np.abs(out[1]).max() < 1e-9    # one rounding further: outside
    assert within > 0


@pytest.mark.parametrize("linear", [False, True])
def test_weights_at_exactly_one_localisation_distance(linear, monkeypatch):
    """The two polynomials of the taper differ by 6e-7 at ri = 1 (their REAL(4) literals); the
    side is that of the quotient distance / local_dist, for local_dist within two roundings
    of the distance of a column from an observation.  The expected distance is formed by the
    reference's operations with the GPU's cos, sin and acos."""
    import torch
    import letkf_gb300 as lg
    import synth
    if linear:
        monkeypatch.setenv("LETKF_GB300_LINEAR_SEARCH", "1")
    base = lg.preset("tiny2d").replace(n_obs=1)
    w = synth.make_workload(base)
    lat, lon = lg.model_grid(base)
    w.obs.lat[:], w.obs.lon[:] = 12.34375, 100.71875
    pi = float(np.float32(3.14159274101257324))
    earth = float(np.float32(6371.393))
    rad = lambda x: torch.tensor(x / 180.0 * pi, dtype=torch.float64, device="cuda")  # noqa: E731
    x1, y1 = rad(12.34375), rad(100.71875)

    def taper(ri):
        if ri > 1.0:
            rj = (ri / 12.0 - 0.5) * ri + 0.625
            rj = rj * ri + float(np.float32(1.666667))
            return (rj * ri - 5.0) * ri + 4.0 - float(np.float32(0.6666667)) / ri
        rj = (-0.25 * ri + 0.5) * ri + 0.625
        return (rj * ri - float(np.float32(1.666667))) * (ri * ri) + 1.0

    other = 0
    for i, j in ((9, 11), (11, 10), (8, 9), (12, 12), (10, 8), (10, 13)):
        x2, y2 = rad(float(lat[i])), rad(float(lon[j]))
        v = torch.cos(x1) * torch.cos(x2) * torch.cos(y1 - y2) + torch.sin(x1) * torch.sin(x2)
        angle = float(torch.acos(v))
        dist = earth * angle
        col = j * base.num_lat + i
        for step in (-2, -1, 0, 1, 2):
            ld = dist
            for _ in range(abs(step)):
                ld = float(np.nextafter(ld, np.inf if step > 0 else 0.0))
            ctx = lg.Letkf(base.replace(local_dist=ld))
            ctx.set_obs(w.obs)
            xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
            ctx.letkf_run(0, w.xb, w.axb, xa, axa)
            _, rloc = ctx.column_list(col)
            ctx.letkf_final()
            assert rloc.size == 1
            assert abs(rloc[0] - taper(dist / ld)) < 1e-13, (i, j, step)
            other += (angle * (earth / ld) > 1.0) != (dist / ld > 1.0)
    assert other > 0  # the product with the rounded reciprocal would take the other side


@pytest.mark.parametrize("name,ens", [("tiny3d", 16), ("small3d", 40), ("tiny3d", 64)])
def test_wait_limit_reports_timeout_and_context_recovers(name, ens):
    """A wait limit of 1 ns makes the first wait between the FP64 Gram's roles run out: every
    role leaves, the issuing warp waits (with its full bound) for its own MMAs, the CTAs free
    their tensor memory and return, and the analysis reports LG_ERR_TIMEOUT.  With the
    default limit back the same context's next analysis is a fresh context's bit for bit."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset(name).replace(ens=ens)
    w = synth.make_workload(cfg)
    xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
    ctx = lg.Letkf(cfg)
    ctx.set_obs(w.obs)
    ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    want = xa.copy(), axa.copy()
    ctx.letkf_final()
    ctx = lg.Letkf(cfg)
    ctx.set_obs(w.obs)
    ctx.set_wait_limit(1)
    with pytest.raises(RuntimeError, match="LG_ERR_TIMEOUT"):
        ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    ctx.set_wait_limit(0)
    ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    ctx.letkf_final()
    assert np.array_equal(xa, want[0]) and np.array_equal(axa, want[1])


def test_core_reports_an_expired_wait(monkeypatch):
    """An expired wait of the Gram is LG_ERR_TIMEOUT however many of the matrices that it left
    unwritten the transform then finds not to be finite, and lg_letkf_core leaves its
    outputs alone."""
    import torch
    import letkf_gb300 as lg
    L = lg.load_library()
    rng = np.random.default_rng(11)
    cases = [_case(rng, 40, 200) for _ in range(60)]
    nan = [(np.full_like(c[0], np.nan), *c[1:]) for c in cases]
    want = _batch(cases, 1.05)
    st, *_ = _batch(nan, 1.05)  # leaves NaN matrices behind in the core's memory
    assert st == LG_ERR_EIG
    monkeypatch.setenv("LETKF_GB300_WAIT_NS", "1")
    st, *_ = _batch(cases, 1.05)
    assert st == -11
    trans, wbar = np.full((40, 40), 7.0), np.full(40, 7.0)
    hx, rd, dep, rloc = cases[0]
    P = lambda a, t=C.c_double: a.ctypes.data_as(C.POINTER(t))  # noqa: E731
    assert L.lg_letkf_core(40, 200, P(hx), P(rd, C.c_float), P(dep), P(rloc), P(trans), P(wbar),
                           1.05) == -11
    assert (trans == 7.0).all() and (wbar == 7.0).all()
    monkeypatch.delenv("LETKF_GB300_WAIT_NS")
    got = _batch(cases, 1.05)
    assert got[0] == 0 and np.array_equal(got[1], want[1]) and np.array_equal(got[2], want[2])
    torch.cuda.synchronize()


def test_first_call_of_a_process_on_a_stream_of_its_own():
    """The node table is on the device before the first launch that reads it, also where that
    is on a non-blocking stream, which is not ordered after the upload's: a process's first
    core call equals its second."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    code = (
        "import sys, ctypes as C; sys.path[:0] = [%r, %r]\n"
        "import torch, letkf_gb300 as lg\n"
        "L = lg.load_library(); k, nb = 16, 2000\n"
        "s = torch.cuda.Stream()\n"
        "n = torch.zeros(nb, dtype=torch.int32).cuda(); off = n.long()\n"
        "tr = [torch.zeros((nb, k, k), dtype=torch.float64).cuda() for _ in range(2)]\n"
        "wb = torch.zeros((nb, k), dtype=torch.float64).cuda(); torch.cuda.synchronize()\n"
        "P = lambda x: C.c_void_p(x.data_ptr())\n"
        "for t in tr:\n"
        "    assert L.lg_core_batch(k, nb, P(n), P(off), None, None, None, None, 1.05, 0, P(t), P(wb),\n"
        "                           C.c_void_p(s.cuda_stream)) == 0\n"
        "torch.cuda.synchronize()\n"
        "assert torch.equal(*tr) and abs(float(tr[0][0, 0, 0]) - 1.05 ** 0.5) < 1e-14\n"
        % (os.path.dirname(here), os.path.join(os.path.dirname(here), "dida-thhpca_gb300")))
    for _ in range(3):
        subprocess.run([sys.executable, "-c", code], check=True, timeout=120)


def test_core_calls_from_several_threads_and_streams():
    """Calls of different sizes on four threads, each with its own stream, share the kernels'
    shared-memory limits and the memory pool and
    give the results of calls one after another."""
    import threading
    import torch
    import letkf_gb300 as lg
    L = lg.load_library()
    rng = np.random.default_rng(77)
    jobs = []
    for k, nb in ((40, 300), (64, 40), (9, 900), (96, 60)):
        base = [_case(rng, k, p) for p in (0, 5, 3 * k)]
        cases = [base[i % 3] for i in range(nb)]
        want = _batch(cases, 1.05)
        n = np.array([c[0].shape[0] for c in cases], np.int32)
        off = np.concatenate([[0], np.cumsum(n)[:-1]]).astype(np.int64)
        dev = [torch.from_numpy(a).cuda() for a in (n, off)]
        dev += [torch.from_numpy(np.concatenate([c[i] for c in cases])).cuda() for i in range(4)]
        outs = [torch.zeros((nb, k, k), dtype=torch.float64, device="cuda"),
                torch.zeros((nb, k), dtype=torch.float64, device="cuda")]
        jobs.append((k, nb, dev, outs, want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    P = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    bad = []

    def work(k, nb, dev, outs, want, s):
        torch.cuda.set_device(0)
        for _ in range(20):
            st = L.lg_core_batch(k, nb, *[P(d) for d in dev], 1.05, 0, P(outs[0]), P(outs[1]),
                                 C.c_void_p(s.cuda_stream))
            if st != 0:
                bad.append((k, st))
                return
            with torch.cuda.stream(s):
                got = [o.cpu().numpy() for o in outs]
            if not all(np.array_equal(a, b) for a, b in zip(got, want[1:])):
                bad.append(k)
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_core_workspace_is_given_back():
    """A call that needed more than the pool keeps (64 MiB) returns the rest to the device
    before it returns itself."""
    import torch
    import letkf_gb300 as lg
    L = lg.load_library()
    k, nb = 64, 8192  # 276 MB of workspace
    n = torch.zeros(nb, dtype=torch.int32, device="cuda")
    off = torch.zeros(nb, dtype=torch.int64, device="cuda")
    tr = torch.zeros((nb, k, k), dtype=torch.float64, device="cuda")
    wb = torch.zeros((nb, k), dtype=torch.float64, device="cuda")
    P = lambda x: C.c_void_p(x.data_ptr())  # noqa: E731
    s = torch.cuda.Stream()
    for stream in (None, C.c_void_p(s.cuda_stream)):
        for count in (64, nb):  # the small call first: kernels loaded, pool begun
            before = torch.cuda.mem_get_info()[0]
            assert L.lg_core_batch(k, count, P(n), P(off), None, None, None, None, 1.05, 0, P(tr),
                                   P(wb), stream) == 0
            held = before - torch.cuda.mem_get_info()[0]
        assert held <= 72 << 20


def test_default_chunk_falls_back_to_one_gib(monkeypatch):
    """Above 104 members the default chunk is larger than 1 GiB of Gram matrices; where its
    workspace cannot be had, the analysis runs in chunks of 1 GiB as before.  At 128 members
    12 288 solves need 4.8 GB of rotation log per stream, 8192 need 3.2: 4000 MiB lies between."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset("tiny3d").replace(ens=128, num_lat=24, num_lon=48, nz=12,
                                      precision=lg.LG_PREC_MIXED)  # 13 824 solves
    w = synth.make_workload(cfg)
    out = []
    for limited in (False, True):
        ctx = lg.Letkf(cfg)
        assert ctx.tuning()["chunk_mb"] > 1024
        ctx.set_obs(w.obs)
        if limited:
            monkeypatch.setenv("LETKF_GB300_ALLOC_LIMIT_MB", "4000")
        else:
            ctx.set_tuning(chunk_mb=1024)
        xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
        ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        out.append((xa, axa, ctx.stats()["n_chunks"]))
        assert ctx.tuning()["chunk_mb"] == 1024
        if limited:  # a chunk size that the caller asked for is not changed
            ctx.set_tuning(chunk_mb=1536)
            with pytest.raises(RuntimeError, match="LG_ERR_NOMEM"):
                ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        ctx.letkf_final()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][2] == out[1][2] == 2


def test_letkf_core_without_host_memory():
    """lg_letkf_core's host staging block cannot be had (a data limit of the process below
    its 200 MB): LG_ERR_NOMEM, the process goes on, and with the limit lifted the same call
    works."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    code = (
        "import sys, resource; sys.path[:0] = [%r, %r]\n"
        "import numpy as np, torch, letkf_gb300 as lg\n"
        "rng = np.random.default_rng(0)\n"
        "def case(p, k=64):\n"
        "    return rng.standard_normal((p, k)), np.ones(p, np.float32), np.ones(p), np.ones(p)\n"
        "small, big = case(100), case(400_000)\n"
        "lg.letkf_core(*small, 1.05)\n"
        "data = [int(l.split()[1]) for l in open('/proc/self/status') if l.startswith('VmData')][0]\n"
        "lim = resource.getrlimit(resource.RLIMIT_DATA)\n"
        "resource.setrlimit(resource.RLIMIT_DATA, ((data << 10) + (64 << 20), lim[1]))\n"
        "try:\n"
        "    lg.letkf_core(*big, 1.05); st = 'no error'\n"
        "except RuntimeError as e:\n"
        "    st = str(e)\n"
        "resource.setrlimit(resource.RLIMIT_DATA, lim)\n"
        "t, w = lg.letkf_core(*big, 1.05)\n"
        "assert np.isfinite(t).all() and np.isfinite(w).all()\n"
        "print(st)\n"
        % (os.path.dirname(here), os.path.join(os.path.dirname(here), "dida-thhpca_gb300")))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-500:]
    assert "LG_ERR_NOMEM" in r.stdout


def test_entries_of_solves_redone_in_fp64_count_once():
    """Ensemble rows below 2^-400 send every solve to the FP64 kernel; lg_stats counts its
    entries once."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset("tiny2d").replace(ens=16)
    w = synth.make_workload(cfg)
    n = []
    for scale in (1.0, 2.0 ** -450):
        ctx = lg.Letkf(cfg)
        ctx.set_obs(w.obs)
        xb, axb = w.xb * scale, w.axb * 0.0  # (a mean would round the spread away in H(x))
        xa, axa = np.zeros_like(xb), np.zeros_like(axb)
        ctx.letkf_run(0, xb, axb, xa, axa)
        yb, _ = ctx.hx(ctx.stats()["n_entries"])
        n.append(ctx.stats()["n_gram_entries"])
        ctx.letkf_final()
        assert 0.0 < np.abs(yb).max() < 100.0 * scale
    assert n[0] > 0 and n[0] == n[1]


@pytest.mark.parametrize("k", [24, 40, 41, 64])
def test_a_later_chunk_left_to_the_fp64_kernel(k):
    """A list whose second chunk (896 kept entries make one) has values below 2^-400 after
    the first has been written: the whole solve is redone.  With a NaN there, the solve
    fails and its neighbours do not."""
    rng = np.random.default_rng(60 + k)
    good, late, nan = _case(rng, k, 1500), list(_case(rng, k, 1500)), list(_case(rng, k, 1500))
    late[0] = late[0].copy()
    late[0][896:] *= 2.0 ** -450
    nan[0] = nan[0].copy()
    nan[0][1300, 2] = np.nan
    st, tr, wb = _batch([good, tuple(late), good], 1.05)
    assert st == 0
    for c, t, w in zip((good, late, good), tr, wb):
        t0, w0 = _reference(*c, 1.05)
        assert np.allclose(t, t0, rtol=1e-11, atol=1e-11)
        assert np.allclose(w, w0, rtol=1e-11, atol=1e-11)
    st, tr2, wb2 = _batch([good, tuple(nan), good], 1.05)
    assert st == LG_ERR_EIG and np.isnan(tr2[1]).all()
    for i in (0, 2):
        assert np.array_equal(tr2[i], tr[i]) and np.array_equal(wb2[i], wb[i])


@pytest.mark.parametrize("k", [9, 33, 40])
def test_core_lanes_by_launch_size(k):
    """Launches of 30, 100, 225, 900 and 6500 warps of vectors: 8, 4, 2, 1 and 1 lanes per
    vector in the matrix kernel, 8, 8, 4, 2 and 1 in the reflections.  A solve's result does
    not depend on the launch it is in."""
    rng = np.random.default_rng(k)
    base = [_case(rng, k, p) for p in (0, 5, 3 * k, 2)]
    first = None
    for warps in (30, 100, 225, 900, 6500):
        nb = warps * 32 // k
        st, tr, wb = _batch([base[i % 4] for i in range(nb)], 1.05)
        assert st == 0
        if first is None:
            first = tr[:4], wb[:4]
            for c, t, w in zip(base, tr, wb):
                _check(c, 1.05, t, w)
        for i in range(4):
            assert (tr[i::4] == first[0][i]).all() and (wb[i::4] == first[1][i]).all()


@pytest.mark.parametrize("nz,vcoord", [(7, 0), (8, 0), (32, 0), (8, 1), (300, 0)])
def test_observations_at_and_around_half_levels(nz, vcoord):
    """Observations exactly on a half level, one and a few roundings (FP64 and FP32) beside
    it, above the top and below the ground: nz = 7 and 8 around the line from which the
    levels are passed in FP32, 300 beyond the 256 levels that are.  H(x) against the
    oracle's with the tolerance of the other H(x) tests, and every profile's levels both
    ascending and descending (the search index persists)."""
    import letkf_gb300 as lg
    import synth
    from oracle import oracle as orc
    cfg = lg.preset("tiny3d").replace(nz=nz, vcoord=vcoord, ens=33, n_obs=10)
    w = synth.make_workload(cfg)
    w.xb[:, :, 0] = 0.0
    w.axb[:, :, 0] = 98765.0
    # temperatures that jump between levels, so that a wrong level shows
    rng = np.random.default_rng(nz)
    w.axb[:, :, 1:] += 50.0 * rng.standard_normal(w.axb[:, :, 1:].shape)
    a, b, p0, ptop = lg.vertical_coord(cfg)
    if vcoord == lg.LG_VCOORD_SIGMA:
        lev = a * (98765.0 - ptop) + ptop
    else:
        lev = a * (p0 - ptop) + b * (98765.0 - ptop) + ptop
    half = 0.5 * (lev[1:] + lev[:-1])
    ph = [half, half * (1 + 2.0 ** -52), half * (1 - 2.0 ** -52), half * (1 + 2.0 ** -24),
          half * (1 - 2.0 ** -24), half * (1 + 1e-6), half * (1 - 1e-6), [1.0, 2e5]]
    ph = np.concatenate(ph)
    n, onz = 400, 4
    ph = rng.choice(ph, (n, onz))
    ph[::2].sort(axis=1)
    lat, lon = synth.obs_locations(cfg, rng, n)
    obs = lg.ObsSet([(onz, 2, [1, 3])], np.zeros(n, np.int32), lat, lon, ph.ravel(),
                    rng.standard_normal(n * onz * 2), np.ones(n * onz * 2))
    ctx = lg.Letkf(cfg)
    ctx.set_obs(obs)
    xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
    ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    o = orc.Oracle(cfg, obs)
    yb_o, dis_o, _ = o.hx(w.xb, w.axb)
    yb, dis = ctx.hx(o.n_entries)
    ctx.letkf_final()
    assert np.allclose(yb, yb_o, rtol=1e-12, atol=1e-12 * np.abs(yb_o).max())
    assert np.allclose(dis, dis_o, rtol=1e-12, atol=1e-12 * np.abs(dis_o).max())


@pytest.mark.parametrize("nz,ens", [(5, 16), (5, 33), (8, 33), (24, 16), (24, 33)])
def test_analysis_lanes_by_launch_size(nz, ens, monkeypatch):
    """Analyses of 500, 800 and 2400 warps of vectors: 4, 2 and 1 lanes per vector in the
    solves, 8, 4 and 2 in the reflections (2-D analyses of this grid: 8 and 8), against the
    QL route (a sweep limit below the default selects it) with the path's tolerance."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset("tiny3d").replace(nz=nz, ens=ens)
    w = synth.make_workload(cfg)
    out = []
    for limit in (None, "59"):
        if limit:
            monkeypatch.setenv("LETKF_GB300_QL_ITERS", limit)
        ctx = lg.Letkf(cfg)
        ctx.set_obs(w.obs)
        xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
        ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        assert (ctx.stats()["ms_ql"] > 0.1) == bool(limit)  # the two routes
        ctx.letkf_final()
        out.append(xa + axa[..., None])
    i = slice(cfg.halo, -cfg.halo)
    inc = np.abs(out[1] - (w.xb + w.axb[..., None]))[i, i].max()
    assert np.abs(out[0] - out[1])[i, i].max() <= 1e-10 * inc


def test_rotation_log_overflow_above_64_members(monkeypatch):
    """96 members take the QL route: with a log of one octet every solve overflows and is
    redone by the accumulating solver, whose rounding differs from the replay's."""
    out = []
    for cap in (None, "5"):
        if cap:
            monkeypatch.setenv("LETKF_GB300_ROT_CAP", cap)
        cfg, w, ctx, o, got, ref = _run_both("tiny3d", ens=96)
        assert _rel_err(cfg, w, got, ref[:2]) < RTOL_ANALYSIS
        assert ctx.stats()["n_eig_fail"] == 0
        ctx.letkf_final()
        out.append(got[0][cfg.halo:-cfg.halo, cfg.halo:-cfg.halo])
    differ = (out[0] != out[1]).any(axis=(2, 3))
    assert differ.all()  # in every column


@pytest.mark.parametrize("rho", [1e-300, 1e-12, 1e12, 1e200])
def test_any_inflation(rho):
    """(k - 1) / rho far below or above a full-rank C: W is (C / (k - 1) + I / rho)^(-1/2)."""
    rng = np.random.default_rng(8)
    k, p = 12, 90
    case = (rng.standard_normal((p, k)), np.ones(p, np.float32), rng.standard_normal(p), np.ones(p))
    st, tr, wb = _batch([case], rho)
    assert st == 0
    t0, w0 = _reference(*case, rho)
    assert np.allclose(wb[0], w0, rtol=1e-9, atol=1e-9 * np.abs(w0).max())
    assert np.allclose(tr[0], t0, rtol=1e-9, atol=1e-9 * np.abs(t0).max())


@pytest.mark.parametrize("name,ens", [("tiny3d", 54), ("tiny3d", 55), ("tiny3d", 56), ("tiny2d", 55)])
def test_pairs_factored_at_a_time(name, ens, monkeypatch):
    """With four state rows 32 (solve, node) pairs are factored at a time up to 54 members and
    16 from 55 on: both sides against the QL route, tolerance of the path."""
    from test_gpu_ft import test_analysis_against_the_ql_route as against_ql
    against_ql(name, ens, monkeypatch)
