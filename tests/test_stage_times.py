"""Stage times count the whole convolution as G2G.  On a large grid with few
points slot 1 is one launch that copies a grid of 250 KB, slot 3 one launch that
gathers 2,000 points, and the transforms along x, the larger half of the
convolution, take longer than both together: slot 1 stays near slot 3.
"""
import numpy as np
import pytest

from conftest import make_problem

pytestmark = pytest.mark.gpu


def test_transforms_along_x_belong_to_the_convolution():
    import sgtsne_b200 as S
    rp, col, val, _ = make_problem(n=2000, dim=20, ncomp=5, k=12, seed=3)
    y0 = np.random.default_rng(3).uniform(-43.0, 43.0, (2000, 2)).astype(np.float32)
    p = S.default_params(d=2, format=S.FORMAT_CSR, max_iter=24, alpha=1.0, h=0.7,
                         grid_mode=S.GRID_FIXED, ng=124)
    ctx = S.Context(0)
    try:
        job = S.Job(ctx, p, rp, col, val.astype(np.float32), device_mem=False)
        job.set_y(y0, S.LAYOUT_POINT_MAJOR, False)
        t = np.zeros(7003)
        job.run_timed(24, t)
        assert job.info().grid_points == 126
        job.close()
    finally:
        ctx.close()
    t = np.median(t[:7 * 24].reshape(24, 7)[4:], 0)
    print("\nstage ms:", np.round(t, 4))
    assert 0 < t[1] < 1.2 * t[3] < t[2]
