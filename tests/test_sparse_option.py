"""curig_opts.sparse sets the spreader's threshold; the interpolator keeps its own
(DEFAULT_SPARSE_I, 16).  Shown by the tile-load hook: with loads that are never
issued, an interpolator on its tiles reports the wait that ran out, one that reads
the grid directly has nothing to wait for.  Crowded bins, so that every chunk
holds more than 16 visibilities but fewer than a large `sparse`.

And the interpolator's direct reads against its tiles (its threshold from
curig_test_sparse_interp): the same kw^3 products per visibility in another
order, FP32 2e-6 and FP64 1e-13 of the norm."""
import numpy as np
import pytest

from conftest import disk_inputs

pytestmark = pytest.mark.gpu


def _plan(precision, nx, ny, eps, uvw, freq, **kw):
    import torch
    from curig_b200 import GridderPlan
    fov = 2.0 * np.pi / 180
    p = GridderPlan(1, nx, ny, fov / nx, fov / ny, eps, 2.0, -1, precision=precision, **kw)
    p.setpts(torch.from_numpy(np.ascontiguousarray(uvw)).cuda(), freq)
    return p


@pytest.mark.parametrize("precision,eps", [("fp32", 1e-5), ("fp64", 1e-8)])
@pytest.mark.parametrize("sparse", [128, 1 << 30, 0, -1])
def test_sparse_is_the_spreaders(precision, eps, sparse):
    import torch

    import curig_b200._lib as L
    n, nrow = 256, 20000
    freq, uvw, ms, wgt = disk_inputs(nrow, 1, n, 2.0, max_pix=30.0, wmax=20.0, seed=41)
    ct = torch.complex64 if precision == "fp32" else torch.complex128
    img = torch.ones((n, n), dtype=ct, device="cuda")
    vis = torch.empty((nrow, 1), dtype=ct, device="cuda")
    L.lib.curig_test_tile_wait(64, 1)
    try:
        p = _plan(precision, n, n, eps, uvw, freq, sparse=sparse)
        p.execute_dir(2, vis, None, img)
        with pytest.raises(L.CurigError) as err:
            p.status()
    finally:
        L.lib.curig_test_tile_wait(0, 0)
    assert err.value.code == 4
    p.close()


@pytest.mark.parametrize("precision,eps", [("fp32", 2e-1), ("fp32", 1e-5), ("fp32", 1e-6), ("fp64", 1e-4),
                                           ("fp64", 1e-9), ("fp64", 1e-11)])
@pytest.mark.parametrize("nx,ny,opts", [(64, 64, {}), (75, 53, {}), (64, 48, {"w_term": 1}), (64, 64, {"bin_z": 2}),
                                        (49, 64, {"bin_xy": 5})])
def test_direct_reads_match_tiles(precision, eps, nx, ny, opts):
    import torch

    import curig_b200._lib as L
    freq, uvw, ms, wgt = disk_inputs(700, 3, min(nx, ny), 2.0, f0=0.9e9, fmax=1.1e9, max_pix=0.49 * min(nx, ny),
                                     wmax=400.0, seed=5)
    ct = torch.complex64 if precision == "fp32" else torch.complex128
    img = torch.from_numpy(np.random.default_rng(6).standard_normal((nx, ny)) + 0j).to(ct).cuda()
    out = {}
    try:
        for sparse in (0, 1 << 30, 3):
            L.lib.curig_test_sparse_interp(sparse)
            p = _plan(precision, nx, ny, eps, uvw, freq, **opts)
            v = torch.empty(ms.shape, dtype=ct, device="cuda")
            p.execute_dir(2, v, None, img)
            p.status()
            out[sparse] = v.cpu().numpy()
            p.close()
    finally:
        L.lib.curig_test_sparse_interp(-1)
    tol = 2e-6 if precision == "fp32" else 1e-13
    for sparse in (1 << 30, 3):
        assert np.linalg.norm(out[sparse] - out[0]) < tol * np.linalg.norm(out[0])
