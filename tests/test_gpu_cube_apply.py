"""Fixed-point application of the cube solves (lg_cube.cu): ensemble sizes that
do not fill a batch of rows or a warp, level groups with a short last group, and
overlapping cubes, against the oracle at the cube analyses' tolerance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ens", [2, 3, 7, 31, 33, 64, 65, 100, 128])
@pytest.mark.parametrize("name,over", [("tiny2d", dict(cube_n=3, overlap=1)),
                                       ("tiny3d", dict(cube_n=2, cube_nz=3))])
def test_ensemble_sizes(name, over, ens):
    import letkf_gb300 as lg
    import synth
    from test_gpu_cubes import _oracle, _rel_err
    cfg = lg.preset(name).replace(ens=ens, **over)
    w = synth.make_workload(cfg)
    xa_o, axa_o, _ = _oracle(cfg, w)
    ctx = lg.Letkf(cfg)
    ctx.set_obs(w.obs)
    xa, axa = np.zeros_like(w.xb), np.zeros_like(w.axb)
    ctx.letkf_run(0, w.xb, w.axb, xa, axa)
    assert ctx.stats()["n_eig_fail"] == 0
    assert _rel_err(cfg, w, (xa, axa), (xa_o, axa_o)) < 1e-10
    h = cfg.halo
    scale = np.abs(xa_o).max()
    assert np.abs(xa[h:-h, h:-h].sum(axis=-1)).max() <= 1e-13 * ens * scale
    ctx.letkf_final()
