"""The bounds-checked build (test_bounds_check.py) over the paths that depend on
the size of the call and of the grid: binning by ranks and by cursors (which large
calls take; curig_test_ranked_bytes lets small ones take them), with one and three
row slabs; the row passes of every form (units that interleave or not, rows in
two halves, partial windows of the grid, odd images) and the library's rows beside
them; the third axis of the 3-D transform; the general tile kernels; the
interpolator's direct reads alone and not at all (curig_test_sparse_interp).

The checked build must raise no flag and agree with the regular one: the order of
the grid's additions differs, 1e-12 of the norm (FP64) and 1e-5 (FP32, as there)."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CHECK_LIB = os.path.join(ROOT, "curig_b200", "libcurafft_check.so")
sys.path.insert(0, HERE)

from conftest import disk_inputs, l2err  # noqa: E402

BINNING = [(prec, nchan, slabs, limit) for prec in (0, 1) for nchan in (1, 3) for slabs in (1, 3) for limit in (0, -1)]
# image, grid (nxdirty's axis, nydirty's axis; w-free; None: the size rule with the
# w axis), largest |u|, |v| in cycles per pixel, options
GRIDS = [((64, 64), None, 0.2, {}), ((75, 53), None, 0.49, {}), ((33, 40), None, 0.3, {"bin_z": 2}),
         ((16, 20), (40, 48), 0.5, {}), ((15, 7), (1458, 1500), 0.1, {}), ((31, 20), (4608, 8192), 0.3, {}),
         ((16, 21), (6000, 64), 0.2, {}), ((15, 20), (64, 5000), 0.2, {}), ((24, 24), (2916, 4800), 0.3, {}),
         ((16, 16), (10000, 40), 0.2, {}), ((40, 40), None, 0.3, {"eps": 1e-13}),
         ((64, 49), None, 0.49, {"direct": 1 << 30}), ((20, 21), (40, 48), 0.49, {"direct": 1 << 30}),
         ((64, 49), None, 0.49, {"direct": 0, "bin_z": 2})]
MODES = [(12, 10, 8), (31, 17, 40), (9, 20, 130)]


def binning(L, prec, nchan, slabs, limit):
    n, nrow = 64, 4000
    px = 2.0 * np.pi / 180 / n
    freq, uvw, ms, wgt = disk_inputs(nrow, nchan, n, 2.0, f0=0.9e9, fmax=1.1e9, max_pix=31.0, wmax=300.0, seed=51)
    ct, rt = (np.complex64, np.float32) if prec else (np.complex128, np.float64)
    uvw, ms, wgt = np.ascontiguousarray(uvw), ms.astype(ct), np.ascontiguousarray(wgt.astype(rt))
    img = (np.random.default_rng(52).standard_normal((n, n)) + 0j).astype(ct)
    o = L.make_opts(precision=prec, accumulate=3, slabs=slabs)
    d, v = np.zeros((n, n), dtype=ct), np.zeros_like(ms)
    L.lib.curig_test_ranked_bytes(limit)
    try:
        l0 = L.lib.curig_launch_count()
        L.check(L.lib.curig_ms2dirty(nrow, nchan, n, n, px, px, freq.ctypes.data, uvw.ctypes.data, ms.ctypes.data,
                                     wgt.ctypes.data, d.ctypes.data, 1e-5, 2.0, -1, ctypes.byref(o)), "ms2dirty")
        launches = L.lib.curig_launch_count() - l0
        L.check(L.lib.curig_dirty2ms(nrow, nchan, n, n, px, px, freq.ctypes.data, uvw.ctypes.data, v.ctypes.data,
                                     wgt.ctypes.data, img.ctypes.data, 1e-5, 2.0, -1, ctypes.byref(o)), "dirty2ms")
    finally:
        L.lib.curig_test_ranked_bytes(-1)
    return d, v, np.array([launches])


def planes(L, prec, image, grid, reach, opts):
    import torch
    from curig_b200 import GridderPlan
    ct = torch.complex64 if prec else torch.complex128
    nx, ny = image
    opts = dict(opts)
    eps = opts.pop("eps", 1e-5 if prec else 1e-9)
    direct = opts.pop("direct", -1)               # the interpolator's threshold
    if grid:
        opts.update(w_term=1, grid_x=grid[0], grid_y=grid[1])
    rng = np.random.default_rng(nx + ny)
    px = 1e-3
    freq = np.array([299792458.0])
    uvw = rng.uniform(-1, 1, (900, 3)) * [reach / px, reach / px, 0.0 if grid else 2000.0]
    vis = rng.standard_normal((900, 1)) + 1j * rng.standard_normal((900, 1))
    img = rng.standard_normal((nx, ny)) + 1j * rng.standard_normal((nx, ny))
    p = GridderPlan(1, nx, ny, px, px, eps, precision="fp32" if prec else "fp64", accumulate=3, **opts)
    L.lib.curig_test_sparse_interp(direct)
    try:
        p.setpts(torch.from_numpy(uvw).cuda(), freq)
    finally:
        L.lib.curig_test_sparse_interp(-1)
    d = torch.empty((nx, ny), dtype=ct, device="cuda")
    v = torch.empty((900, 1), dtype=ct, device="cuda")
    p.execute_dir(1, torch.from_numpy(vis).to(ct).cuda(), None, d)
    p.execute_dir(2, v, None, torch.from_numpy(img).to(ct).cuda())
    p.status()
    out = d.cpu().numpy(), v.cpu().numpy()
    p.close()
    return out


def volume(L, prec, modes):
    import torch
    ct = torch.complex64 if prec else torch.complex128
    rng = np.random.default_rng(sum(modes))
    xyz = [torch.from_numpy(rng.uniform(-np.pi, np.pi, 800)).cuda() for _ in range(3)]
    c = torch.from_numpy(rng.standard_normal(800) + 1j * rng.standard_normal(800)).to(ct).cuda()
    fk = torch.from_numpy(rng.standard_normal(modes) + 1j * rng.standard_normal(modes)).to(ct).cuda()
    out = []
    for kind in (1, 2):
        o = L.make_opts(precision=prec, accumulate=3)
        h = ctypes.c_void_p()
        L.check(L.lib.curig_nufft3d_makeplan(kind, *modes, 1e-5 if prec else 1e-9, 1, 2.0, ctypes.byref(o),
                                             ctypes.byref(h)), "makeplan")
        L.check(L.lib.curig_nufft3d_setpts(h, 800, *[a.data_ptr() for a in xyz]), "setpts")
        a, b = (c, torch.empty_like(fk)) if kind == 1 else (torch.empty_like(c), fk)
        L.check(L.lib.curig_nufft_execute(h, a.data_ptr(), b.data_ptr()), "execute")
        L.check(L.lib.curig_plan_status(h), "status")      # (both handles begin with their plan)
        out.append((b if kind == 1 else a).cpu().numpy())
        L.check(L.lib.curig_nufft_destroy(h), "destroy")
    return tuple(out)


def run_all(L):
    out = {}
    for case in BINNING:
        out["binning %s" % (case,)] = binning(L, *case)
    for prec in (0, 1):
        for case in GRIDS:
            out["planes %d %s" % (prec, case)] = planes(L, prec, *case)
        for modes in MODES:
            out["volume %d %s" % (prec, modes)] = volume(L, prec, modes)
    return {"%s / %d" % (k, i): a for k, arrays in out.items() for i, a in enumerate(arrays)}


def _worker(path):
    sys.path[:0] = [ROOT]
    import curig_b200._lib as L
    assert os.path.samefile(L.LIB_PATH, CHECK_LIB), L.LIB_PATH
    res = run_all(L)                                # a raised flag fails the call or status()
    np.savez(path, names=np.array(list(res)), **{"a%d" % i: a for i, a in enumerate(res.values())})


@pytest.mark.gpu
def test_size_dependent_paths_stay_in_their_buffers(tmp_path):
    import curig_b200._lib as L
    path = str(tmp_path / "checked.npz")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), path], env=dict(os.environ, CURIG_LIB=CHECK_LIB),
                       capture_output=True, text=True, timeout=1200)
    assert r.returncode == 0, r.stderr[-4000:]
    z = np.load(path)
    chk = {str(n): z["a%d" % i] for i, n in enumerate(z["names"])}
    ref = run_all(L)
    assert list(chk) == list(ref)
    for name, a in ref.items():
        tol = 1e-5 if a.dtype == np.complex64 else 1e-12
        assert l2err(a, chk[name]) < tol, (name, l2err(a, chk[name]))


@pytest.mark.gpu
@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 2e-6)])
@pytest.mark.parametrize("nchan", [1, 3])
@pytest.mark.parametrize("slabs", [1, 3])
def test_ranks_and_cursors_agree(prec, tol, nchan, slabs):
    """The same points through both: equal sums in another order (exact tiles);
    the cursors' scatter is one launch more."""
    import curig_b200._lib as L
    ranks, cursors = binning(L, prec, nchan, slabs, -1), binning(L, prec, nchan, slabs, 0)
    assert cursors[2][0] == ranks[2][0] + 1
    assert l2err(ranks[0], cursors[0]) < tol and l2err(ranks[1], cursors[1]) < tol


if __name__ == "__main__":
    _worker(sys.argv[1])
