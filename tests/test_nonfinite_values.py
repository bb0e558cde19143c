"""A visibility, weight or pixel that is not finite shows in the result, whatever
path its chunk takes: every tile form of the spreader, the direct reductions of
sparse chunks, narrow and general kernels.  One bad visibility among 1 to 3000 in
one bin makes the whole image not finite (the transforms spread it), and leaves
the next call's image as it was: equal to a plan's that never met one, up to the
order of its additions (1e-12 FP64, 2e-6 FP32)."""
import numpy as np
import pytest

from conftest import l2err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,eps,tol", [("fp64", 1e-8, 1e-12), ("fp32", 1e-4, 2e-6), ("fp64", 1e-13, 1e-12)])
@pytest.mark.parametrize("accumulate", [0, 1, 2, 3])
@pytest.mark.parametrize("sparse", [0, -1, 1 << 30])
@pytest.mark.parametrize("w_term", [0, 1])
def test_one_bad_visibility(precision, eps, tol, accumulate, sparse, w_term):
    import torch
    from curig_b200 import GridderPlan
    ct, rt = (torch.complex64, torch.float32) if precision == "fp32" else (torch.complex128, torch.float64)
    if w_term and eps < 1e-11:
        pytest.skip("no w-free mode beyond width 12")
    n, px = 32, 1e-3
    freq = np.array([299792458.0])
    for nrow in (1, 40, 100, 3000):
        rng = np.random.default_rng(nrow)
        uvw = np.tile([[0.11 / px, -0.2 / px, 30.0]], (nrow, 1)) + rng.uniform(0, 1, (nrow, 3)) * [1e-2, 1e-2, 1.0]
        vis = torch.from_numpy(rng.standard_normal((nrow, 1)) + 1j * rng.standard_normal((nrow, 1))).to(ct).cuda()
        w = torch.from_numpy(rng.uniform(0.5, 1, (nrow, 1))).to(rt).cuda()
        p = GridderPlan(1, n, n, px, px, eps, precision=precision, accumulate=accumulate, sparse=sparse, w_term=w_term)
        p.setpts(torch.from_numpy(uvw).cuda(), freq)

        def image(v, wt):
            d = torch.zeros((n, n), dtype=ct, device="cuda")
            p.execute_dir(1, v, wt, d)
            p.status()
            return d.cpu().numpy()

        ref = image(vis, w)
        assert np.isfinite(ref).all()
        for bad in (complex(float("nan"), 1.0), complex(1.0, float("nan")), complex(0.0, float("inf")),
                    complex(float("-inf"), 0.0)):
            v = vis.clone()
            v[nrow // 2] = bad
            assert not np.isfinite(image(v, w)).any()
            assert not np.isfinite(image(v, None)).any()
        wb = w.clone()
        wb[nrow - 1] = float("nan")
        assert not np.isfinite(image(vis, wb)).any()
        assert l2err(ref, image(vis, w)) < tol
        img = torch.ones((n, n), dtype=ct, device="cuda")
        img[3, 5] = float("nan")
        o = torch.zeros_like(vis)
        p.execute_dir(2, o, w, img)
        assert not np.isfinite(o.cpu().numpy()).any()
        p.close()
