"""A set points that fails leaves its plan without points, so the plan gives its
device memory back; one that is refused for its arguments leaves the last points
in place.  The plan's grid is 1 GiB (8192^2 FP64 cells, one plane), the margin a
quarter of that; the next valid set points gives a fresh plan's results (the same
kernels on the same data: 1e-12, the order of the grid's additions)."""
import numpy as np
import pytest

from conftest import disk_inputs, l2err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_failed_set_points_gives_its_memory_back(axis):
    import torch

    import curig_b200._lib as L
    from curig_b200 import GridderPlan
    n, nrow = 64, 3000
    px = 2.0 * np.pi / 180 / n
    freq, uvw, ms, wgt = disk_inputs(nrow, 1, n, 2.0, max_pix=25.0, seed=21)
    good = torch.from_numpy(np.ascontiguousarray(uvw)).cuda()
    bad = good.clone()
    bad[nrow // 2, axis] = float("nan")
    vis, w = torch.from_numpy(ms).cuda(), torch.from_numpy(wgt).cuda()
    d = torch.empty((n, n), dtype=torch.complex128, device="cuda")

    def new():
        return GridderPlan(1, n, n, px, px, 1e-6, precision="fp64", w_term=1, grid_x=8192, grid_y=8192)

    def image(p):
        p.setpts(good, freq)
        p.execute(vis, w, d)
        p.status()
        return d.cpu().numpy()

    def free():
        torch.cuda.synchronize()
        assert L.lib.curig_release_memory() == 0
        return torch.cuda.mem_get_info()[0]

    p = new()
    ref = image(p)
    p.close()
    free0 = free()
    p = new()
    image(p)
    assert free() < free0 - (1 << 30)
    with pytest.raises(L.CurigError) as err:
        p.setpts(good, np.array([-1.0]))          # refused: the points stay
    assert err.value.code == 7
    p.nrow, p.nchan = nrow, 1
    d.zero_()
    p.execute(vis, w, d)
    assert l2err(ref, d.cpu().numpy()) < 1e-12
    with pytest.raises(L.CurigError) as err:
        p.setpts(bad, freq)
    assert err.value.code == 7
    assert free() > free0 - (1 << 28)
    with pytest.raises(L.CurigError):
        p.execute(vis, w, d)
    p.status()
    assert l2err(ref, image(p)) < 1e-12
    p.close()
