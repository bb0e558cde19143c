"""Window tables of every degree that curig_set_window takes.  Tables beyond
degree 11 run on the general tile kernels; a degree-11 table with zero leading
coefficients is the same window, so both give the same sums in another order:
1e-12 (FP64), 2e-6 (FP32, exact tiles on the degree-11 side)."""
import ctypes

import numpy as np
import pytest

from conftest import disk_inputs, l2err

pytestmark = pytest.mark.gpu

EPS = 1e-3


def _register(learned, L, W, degree):
    coef = np.zeros((W, degree + 1))
    coef[:, degree - 11:] = learned.table(W, learned.init_params(0))
    learned.clear()
    assert L.lib.curig_set_window(W, degree, np.ascontiguousarray(coef).ctypes.data, EPS) == 0


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-6)])
@pytest.mark.parametrize("W,degree", [(2, 12), (5, 12), (6, 15), (12, 15)])
@pytest.mark.parametrize("opts", [{}, {"w_term": 1}, {"bin_z": 2}])
def test_degrees_beyond_the_tables(precision, tol, W, degree, opts):
    import torch

    import curig_b200._lib as L
    from curig_b200 import GridderPlan, learned
    ct, rt = (torch.complex64, torch.float32) if precision == "fp32" else (torch.complex128, torch.float64)
    nx, ny = 64, 50
    px = 2.0 * np.pi / 180 / nx
    freq, uvw, ms, wgt = disk_inputs(1500, 2, ny, 2.0, f0=0.9e9, fmax=1.1e9, max_pix=0.49 * ny, wmax=400.0, seed=31)
    img = torch.from_numpy(np.random.default_rng(32).standard_normal((nx, ny)) + 0j).to(ct).cuda()
    u, v, w = torch.from_numpy(uvw).cuda(), torch.from_numpy(ms).to(ct).cuda(), torch.from_numpy(wgt).to(rt).cuda()
    res = {}
    try:
        for deg in (11, degree):
            _register(learned, L, W, deg)
            p = GridderPlan(1, nx, ny, px, px, EPS, precision=precision, window="learned", accumulate=3, **opts)
            p.setpts(u, freq)
            assert p.info()["kw"] == W
            d = torch.empty((nx, ny), dtype=ct, device="cuda")
            o = torch.empty_like(v)
            p.execute_dir(1, v, w, d)
            p.execute_dir(2, o, w, img)
            p.status()
            res[deg] = d.cpu().numpy(), o.cpu().numpy()
            p.close()
    finally:
        learned.clear()
    assert l2err(res[11][0], res[degree][0]) < tol
    assert l2err(res[11][1], res[degree][1]) < tol


@pytest.mark.parametrize("precision", [0, 1])
def test_one_shot_with_row_slabs(precision):
    import curig_b200._lib as L
    from curig_b200 import learned
    n, nrow, nchan, W = 64, 3000, 2, 6
    px = 2.0 * np.pi / 180 / n
    freq, uvw, ms, wgt = disk_inputs(nrow, nchan, n, 2.0, f0=0.9e9, fmax=1.1e9, max_pix=28.0, wmax=300.0, seed=33)
    ct, rt = (np.complex64, np.float32) if precision else (np.complex128, np.float64)
    uvw, ms, wgt = np.ascontiguousarray(uvw), ms.astype(ct), np.ascontiguousarray(wgt.astype(rt))
    img = (np.random.default_rng(34).standard_normal((n, n)) + 0j).astype(ct)
    res = {}
    try:
        for deg in (11, 13):
            _register(learned, L, W, deg)
            o = L.make_opts(precision=precision, window=1, accumulate=3, slabs=3)
            d, v = np.zeros((n, n), dtype=ct), np.zeros_like(ms)
            assert L.lib.curig_ms2dirty(nrow, nchan, n, n, px, px, freq.ctypes.data, uvw.ctypes.data, ms.ctypes.data,
                                        wgt.ctypes.data, d.ctypes.data, EPS, 2.0, -1, ctypes.byref(o)) == 0
            assert L.lib.curig_dirty2ms(nrow, nchan, n, n, px, px, freq.ctypes.data, uvw.ctypes.data, v.ctypes.data,
                                        wgt.ctypes.data, img.ctypes.data, EPS, 2.0, -1, ctypes.byref(o)) == 0
            res[deg] = d, v
    finally:
        learned.clear()
    tol = 2e-6 if precision else 1e-12
    assert l2err(res[11][0], res[13][0]) < tol and l2err(res[11][1], res[13][1]) < tol
