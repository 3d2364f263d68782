"""FP64 Gram matrices by exact slices on the tensor cores (lg_gram64_tc.cu).

Sizes where the kernel can go wrong: member counts around its tile limits (row
groups of 8, the 48-member split, the full 64), list lengths around its stages
(64 entries), exact sums (256) and chunks (1536), empty lists, and values it has
to leave to the FP64 kernel (non-finite, or far outside its exponent range).

The yardstick is numpy's FP64 evaluation.  Its own rounding and the kernel's
are each some 1e-16 of C's largest element per entry and random, C's condition
number is below 1e4 here, so trans and overline_w agree to about 1e-12; the
repository's tolerance for the batched core, 1e-11, leaves a factor of ten.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LG_ERR_EIG = -7


def _case(rng, k, p):
    hx = rng.standard_normal((p, k))
    hx -= hx.mean(axis=1, keepdims=True)
    rd = (1.0 / rng.uniform(0.5, 2.0, p) ** 2).astype(np.float32)
    return hx, rd, rng.standard_normal(p), rng.uniform(0.0, 1.0, p)


def _reference(hx, rd, dep, rloc, rho):
    k = hx.shape[1]
    rr = np.sqrt(rd.astype(np.float64) * rloc)
    z = hx * rr[:, None]
    lam, v = np.linalg.eigh(z.T @ z)
    lam = lam + (k - 1) / rho
    wbar = v @ ((v.T @ (z.T @ (rr * dep))) / lam)
    w = (v * np.sqrt((k - 1) / lam)) @ v.T
    return (w + wbar[:, None]).T, wbar


def _batch(cases, rho):
    """lg_core_batch (plain FP64) of several solves -> status, trans, overline_w."""
    import torch
    import letkf_gb300 as lg
    L = lg.load_library()
    k, nb = cases[0][0].shape[1], len(cases)
    n = np.array([c[0].shape[0] for c in cases], np.int32)
    off = np.concatenate([[0], np.cumsum(n)[:-1]]).astype(np.int64)
    dev = [torch.from_numpy(np.concatenate([c[i] for c in cases])).cuda() for i in range(4)]
    tn, to = torch.from_numpy(n).cuda(), torch.from_numpy(off).cuda()
    tr = torch.zeros((nb, k, k), dtype=torch.float64, device="cuda")
    wb = torch.zeros((nb, k), dtype=torch.float64, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    st = L.lg_core_batch(k, nb, ptr(tn), ptr(to), *[ptr(t) for t in dev], rho, 0, ptr(tr), ptr(wb),
                         None)
    torch.cuda.synchronize()
    return st, tr.cpu().numpy(), wb.cpu().numpy()


@pytest.mark.parametrize("k", [2, 7, 8, 9, 16, 33, 47, 48, 49, 63, 64])
def test_members_and_list_lengths(k):
    rng = np.random.default_rng(100 + k)
    sizes = [0, 1, 63, 64, 65, 255, 256, 257, 1535, 1536, 1537, 3200]
    cases = [_case(rng, k, p) for p in sizes]
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    for c, t, w, p in zip(cases, tr, wb, sizes):
        t0, w0 = _reference(*c, 1.05)
        assert np.allclose(t, t0, rtol=1e-11, atol=1e-11), p
        assert np.allclose(w, w0, rtol=1e-11, atol=1e-11), p


def test_wide_range_of_weights_and_rows():
    """Rows and weights spread over many binades within one list."""
    rng = np.random.default_rng(5)
    k, p = 40, 700
    hx, rd, dep, rloc = _case(rng, k, p)
    hx *= 2.0 ** rng.integers(-40, 3, p)[:, None]
    rloc *= 2.0 ** rng.integers(-60, 1, p).astype(np.float64)
    rloc[::7] = 0.0
    hx[::11] = 0.0
    st, tr, wb = _batch([(hx, rd, dep, rloc)], 1.1)
    assert st == 0
    t0, w0 = _reference(hx, rd, dep, rloc, 1.1)
    assert np.allclose(tr[0], t0, rtol=1e-11, atol=1e-11)
    assert np.allclose(wb[0], w0, rtol=1e-11, atol=1e-11)


def test_values_left_to_the_fp64_kernel():
    """A NaN row spoils its own solve only; a solve whose magnitudes lie below
    2^-400 gives trans = sqrt(rho) I to rounding (its C vanishes beside
    (k - 1) / rho), and its overline_w keeps its relative accuracy."""
    rng = np.random.default_rng(9)
    k = 24
    good, bad, tiny = _case(rng, k, 300), list(_case(rng, k, 200)), list(_case(rng, k, 150))
    bad[0] = bad[0].copy()
    bad[0][77, 3] = np.nan
    tiny[0] = tiny[0] * 2.0 ** -450
    st, tr, wb = _batch([good, tuple(bad), tuple(tiny), good], 1.05)
    assert st == LG_ERR_EIG
    t0, w0 = _reference(*good, 1.05)
    for i in (0, 3):
        assert np.allclose(tr[i], t0, rtol=1e-11, atol=1e-11)
        assert np.allclose(wb[i], w0, rtol=1e-11, atol=1e-11)
    assert np.isnan(tr[1]).all()
    assert np.allclose(tr[2], np.sqrt(1.05) * np.eye(k), rtol=0, atol=1e-13)
    _, wt = _reference(*tiny, 1.05)
    assert np.allclose(wb[2], wt, rtol=1e-11, atol=0)


@pytest.mark.parametrize("k", [3, 23, 32, 39, 40, 41])
def test_three_slices_per_operand(k):
    """Up to 40 members three slices share an operand's 128 rows and two
    accumulator buffers alternate: list lengths around one to four of the exact
    sums that change them, and weights of one sign (the largest sums)."""
    rng = np.random.default_rng(300 + k)
    sizes = [1, 256, 257, 511, 512, 513, 769, 1025, 1793, 2049]
    cases = [_case(rng, k, p) for p in sizes]
    same = _case(rng, k, 1024)
    same[0][:] = same[0][0] * rng.uniform(0.99, 1.0, 1024)[:, None]  # nearly one row 1024 times
    cases.append(same)
    st, tr, wb = _batch(cases, 1.05)
    assert st == 0
    for c, t, w, p in zip(cases, tr, wb, sizes + ["same"]):
        t0, w0 = _reference(*c, 1.05)
        assert np.allclose(t, t0, rtol=1e-11, atol=1e-11), p
        assert np.allclose(w, w0, rtol=1e-11, atol=1e-11), p
