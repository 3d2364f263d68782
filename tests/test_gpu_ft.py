"""FP64 transform without eigenvalues (lg_ft.cu): W = sqrt(k-1) A^(-1/2) and
overline_w = A^-1 t from shifted tridiagonal solves.

Member counts around a warp's 32 lanes and the ends of the range (7, 64),
spectra from C = 0 to a condition number of 10^9, and analyses with one and four
variables (16 and 6 solves per warp).

Yardstick: numpy's eigh in FP64.  Both it and the kernel are backward stable:
each returns the function of a matrix within about k 2^-53 |A| of A, and a
change E of A moves A^(-1/2) by at most |E| lambda_min^(-3/2) / 2 and A^-1 t by
|E| |t| / lambda_min^2.  The tolerances are those bounds with 8 k 2^-53 |A| for
the two evaluations' |E| together.
"""
import numpy as np
import pytest

from test_gpu_gram64 import _batch, _case

pytestmark = pytest.mark.gpu


def _check(case, rho, trans, wbar):
    hx, rd, dep, rloc = case
    k = hx.shape[1]
    rr = np.sqrt(rd.astype(np.float64) * rloc)
    z = hx * rr[:, None]
    t = z.T @ (rr * dep)
    lam, v = np.linalg.eigh(z.T @ z)
    lam = np.maximum(lam, 0.0) + (k - 1) / rho
    w = (v * np.sqrt((k - 1) / lam)) @ v.T
    wb = v @ ((v.T @ t) / lam)
    err = 8 * k * 2.0 ** -53 * lam.max()
    tol_w = err * 0.5 * np.sqrt(k - 1) * lam.min() ** -1.5 + 1e-14
    tol_b = err * np.linalg.norm(t) / lam.min() ** 2 + 1e-14 * np.abs(wb).max()
    assert np.abs(wbar - wb).max() <= tol_b
    assert np.abs(trans.T - wbar[:, None] - w).max() <= tol_w + 4 * 2.0 ** -53 * np.abs(wbar).max()


@pytest.mark.parametrize("k", [7, 8, 31, 32, 33, 40, 63, 64])
def test_member_counts_and_condition_numbers(k):
    rng = np.random.default_rng(k)
    cases = []
    for scale in (0.0, 1e-9, 1e-3, 1.0, 1e2, 1e4, 1e6):
        for p in (3, 5 * k):  # rank-deficient and full
            hx, rd, dep, rloc = _case(rng, k, p)
            cases.append((hx, (rd * np.float32(scale)).astype(np.float32), dep, rloc))
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    for c, t, w in zip(cases, tr, wb):
        _check(c, 1.05, t, w)


@pytest.mark.parametrize("name,ens", [("tiny2d", 7), ("tiny2d", 33), ("tiny3d", 9), ("tiny3d", 64)])
def test_analysis_against_the_ql_route(name, ens, monkeypatch):
    """The same analysis with the QL route (a sweep limit below the default
    selects it; 59 sweeps still converge) agrees to rounding: the increments
    within 1e-10 of their largest, the repository's tolerance for the path."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset(name).replace(ens=ens)
    w = synth.make_workload(cfg)
    out = []
    for limit in (None, "59"):
        if limit:
            monkeypatch.setenv("LETKF_GB300_QL_ITERS", limit)
        ctx = lg.Letkf(cfg)
        ctx.set_obs(w.obs)
        xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
        ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        ctx.letkf_final()
        out.append(xa + axa[..., None])
    h = cfg.halo
    i = slice(h, -h)
    inc = np.abs(out[1] - (w.xb + w.axb[..., None]))[i, i].max()
    assert np.abs(out[0] - out[1])[i, i].max() <= 1e-10 * inc


@pytest.mark.parametrize("k", [7, 33, 64])
def test_structured_gram_matrices(k):
    """Rows that leave the fixed-point reduction (lg_tri.cu) nothing or little to
    reduce: diagonal, already tridiagonal, zero rows and columns, one dominant
    row, equal rows, and the same at scales far from one."""
    rng = np.random.default_rng(1000 + k)
    eye = np.eye(k)
    tri = eye + np.diag(rng.standard_normal(k - 1), 1)   # z^T z tridiagonal
    hole = rng.standard_normal((3 * k, k))
    hole[:, [0, k // 2, k - 1]] = 0.0
    spike = rng.standard_normal((2 * k, k))
    spike[:, k - 2] *= 1e6
    graded = rng.standard_normal((2 * k, k)) * 2.0 ** -np.arange(k)
    shapes = [eye * rng.uniform(0.5, 2.0, k), tri, hole, spike, graded, graded[:, ::-1],
              np.ones((k, k)), np.outer(np.ones(k), rng.standard_normal(k))]
    cases = []
    for z in shapes:
        for scale in (1.0, 2.0 ** -60, 2.0 ** 12):
            p = z.shape[0]
            cases.append((np.ascontiguousarray(z * scale), np.ones(p, np.float32),
                          rng.standard_normal(p), np.ones(p)))
    st, tr, wb = _batch(cases, 1.1)
    assert st == 0
    for c, t, w in zip(cases, tr, wb):
        _check(c, 1.1, t, w)


@pytest.mark.parametrize("nz", [10, 11, 21, 32])
def test_every_row_in_one_solve(nz, monkeypatch):
    """Without vertical localisation a solve transforms every row of its column:
    31 (a warp with t), 34, 64 and 97 rows (more than a warp), against the QL
    route with the tolerance above."""
    import letkf_gb300 as lg
    import synth
    cfg = lg.preset("tiny3d").replace(nz=nz, vert_dist=-1.0)
    w = synth.make_workload(cfg)
    out = []
    for limit in (None, "59"):
        if limit:
            monkeypatch.setenv("LETKF_GB300_QL_ITERS", limit)
        ctx = lg.Letkf(cfg)
        ctx.set_obs(w.obs)
        xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
        ctx.letkf_run(0, w.xb, w.axb, xa, axa)
        ctx.letkf_final()
        out.append(xa + axa[..., None])
    i = slice(cfg.halo, -cfg.halo)
    inc = np.abs(out[1] - (w.xb + w.axb[..., None]))[i, i].max()
    assert np.abs(out[0] - out[1])[i, i].max() <= 1e-10 * inc


@pytest.mark.parametrize("k,nb", [(7, 1), (9, 3), (40, 1), (41, 100), (64, 70), (40, 400), (33, 700)])
def test_lanes_per_vector(k, nb):
    """Batches from one solve to some hundred: 8, 4, 2 and 1 lanes per vector,
    member counts that leave lanes without elements."""
    rng = np.random.default_rng(17 * k + nb)
    base = [_case(rng, k, p) for p in (0, 5, 3 * k)]
    cases = [base[i % 3] for i in range(nb)]
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    for i in sorted({0, 1, 2, nb // 2, nb - 3, nb - 2, nb - 1} & set(range(nb))):
        _check(cases[i], 1.05, tr[i], wb[i])
    for i in range(3, nb):  # a solve's result does not depend on its place
        assert np.array_equal(tr[i], tr[i % 3]) and np.array_equal(wb[i], wb[i % 3])


@pytest.mark.parametrize("name,ens", [("tiny2d", 56), ("tiny2d", 57), ("tiny3d", 57), ("tiny2d", 64)])
def test_factors_of_half_a_warp(name, ens, monkeypatch):
    """From 57 members on a warp factors 16 (solve, node) pairs at a time, below
    32: both sides of the line against the QL route, tolerance as above."""
    test_analysis_against_the_ql_route(name, ens, monkeypatch)
