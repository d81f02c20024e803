"""Iterations queued before a job has coordinates, alone and in a batch, must
leave the GPU and the job usable: after set_y the job runs as one that was
given coordinates first.  Bar: the repository's for two iterations of a job
against itself (1e-5; sums in L2 differ from run to run).
"""
import numpy as np
import pytest

from conftest import make_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3])
def test_run_before_set_y(d):
    import sgtsne_b200 as S
    rp, col, val, _ = make_problem(n=1500, dim=20, ncomp=5, k=12, seed=d)
    y0 = np.random.default_rng(d).standard_normal((1500, d)).astype(np.float32)
    p = S.default_params(d=d, format=S.FORMAT_CSR, max_iter=8, h={1: 0.5, 2: 0.7, 3: 1.2}[d])
    ctx = S.Context(0)
    try:
        out = []
        for early in (False, True):
            jobs = [S.Job(ctx, p, rp, col, val.astype(np.float32), device_mem=False)
                    for _ in range(2)]
            batch = S.Batch(ctx, jobs, 2)
            if early:
                jobs[0].run(1)
                batch.run(2)
            for j in jobs:
                j.set_y(y0, S.LAYOUT_POINT_MAJOR, False)
            jobs[0].run(2)
            out += [j.get_y(np.empty((1500, d), np.float32), S.LAYOUT_POINT_MAJOR, False, 0)
                    for j in jobs]
            batch.close()
            for j in jobs:
                j.close()
    finally:
        ctx.close()
    assert np.array_equal(out[1], out[3])  # not run since: the coordinates themselves
    assert np.linalg.norm(out[2] - out[0]) <= 1e-5 * np.linalg.norm(out[0])
