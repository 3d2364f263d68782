"""lg_gmcore_to_da_device at the edges of its two forms: one or two members per
thread (odd ensembles, arrays off 16-byte alignment), level counts around the
four loads in flight, one level, and ensembles above a block's 256 threads.
Against the restatement of test_coupler.py, with its tolerances."""
import numpy as np
import pytest

from test_coupler import _restated

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ens,nz,halo,shift", [(1, 1, 1, 0), (2, 1, 1, 0), (7, 5, 1, 0), (64, 33, 1, 0),
                                               (62, 32, 2, 0), (20, 8, 1, 1), (514, 2, 1, 0),
                                               (1023, 1, 1, 0), (16, 4, 0, 0)])
def test_members_levels_and_alignment(ens, nz, halo, shift):
    import torch
    import letkf_gb300 as lg
    nlat, nlon = 5, 6
    rng = np.random.default_rng(ens + nz)
    asub = rng.uniform(0.5, 1.5, (nlat, 2))
    arrays = (rng.normal(1e5, 500, (nlat, nlon, ens)), rng.normal(0, 10, (nz, nlat, nlon, ens)),
              rng.normal(0, 10, (nz, nlat + 1, nlon, ens)), rng.normal(300, 5, (nz, nlat, nlon, ens)),
              asub, asub.sum(axis=1))
    dev = []
    for a in arrays:  # shift: the arrays start 8 bytes after an allocation's start
        buf = torch.empty(a.size + shift, dtype=torch.float64, device="cuda")
        t = buf[shift:].view(a.shape)
        t.copy_(torch.from_numpy(a))
        dev.append(t)
    got = lg.gmcore_to_da(*dev, halo=halo).cpu().numpy()
    ref = _restated(*arrays, halo)
    assert np.array_equal(got[:, :, : 1 + nz], ref[:, :, : 1 + nz])
    assert np.array_equal(got[:, :, 1 + 2 * nz:], ref[:, :, 1 + 2 * nz:])
    v = slice(1 + nz, 1 + 2 * nz)
    assert np.abs(got[:, :, v] - ref[:, :, v]).max() <= 1e-14 * np.abs(ref[:, :, v]).max()
