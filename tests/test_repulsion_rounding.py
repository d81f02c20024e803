"""Repulsive forces at rounding level, where the convolutions take over from
each other, and what they mean for the update inside a batch.

1. Forces of the operator against the FP64 oracle on the same grid, on the grids
   of the plain transforms.  A value is a chain of about 64 + 3 N FP32 sums
   (stencil, transforms, stencil); a random walk of 300 roundings is 1e-6, the
   bar five times that.
2. The update of jobs in a batch, one iteration at a time: from the coordinates
   each iteration starts with, the oracle's dY in FP64 and the rule for the
   gains give the next ones.  A gain may go the other way only where dY or the
   momentum is within rounding of zero (of dY 1e-5 of its root mean square, of
   the momentum what that and the gains make of it), and the step must be the
   rule's for one of the two gains to that error and the coordinates'.
"""
import numpy as np
import pytest

from conftest import make_problem

pytestmark = pytest.mark.gpu

H = {1: 0.5, 2: 0.7, 3: 1.2}
BAR = 5e-6


@pytest.mark.parametrize("d,n,N", [
    (1, 3000, 512), (2, 3000, 16), (2, 3000, 126), (3, 3000, 28), (3, 3000, 33), (3, 3000, 42),
    (3, 3000, 50), (3, 3000, 52), (3, 3000, 72), (3, 60000, 26),
])
def test_forces_at_rounding_level(d, n, N):
    import torch

    import sgtsne_b200 as S
    from oracle import oracle as O
    rng = np.random.default_rng(100 * d + N)
    c = rng.standard_normal((6, d)) * 3
    Y = (c[rng.integers(0, 6, n)] + rng.standard_normal((n, d)) * 0.4).astype(np.float32)
    ctx = S.Context(0)
    try:
        f = torch.empty(n * d, dtype=torch.float32, device="cuda")
        Yd = torch.from_numpy(np.ascontiguousarray(Y)).cuda()
        torch.cuda.synchronize()
        Z, got, _ = ctx.repulsive(n, d, H[d], N - 2, Yd, S.LAYOUT_POINT_MAJOR, f)
        assert got == N
    finally:
        ctx.close()
    Fo, Zo, No, _ = O.repulsive_interp(Y.astype(np.float64), H[d], n1_force=N - 2)
    err = np.linalg.norm(f.cpu().numpy().reshape(n, d) - Fo) / np.linalg.norm(Fo)
    print(f"\n{d}-D, {N} points per axis: force error {err:.2e}, Z {abs(Z - Zo) / abs(Zo):.2e}")
    assert No == N and err <= BAR and abs(Z - Zo) <= BAR * abs(Zo)


def test_gains_of_jobs_in_a_batch(oracle):
    import sgtsne_b200 as S
    jobs, eta = [], 200.0
    ctx = S.Context(0)
    try:
        for i, (n, d, extent) in enumerate([(1200, 2, 24.0), (1500, 3, 20.0), (2500, 2, 40.0),
                                            (1000, 2, 12.0), (2000, 3, 34.0), (1100, 1, 30.0)]):
            rp, col, val, _ = make_problem(n=n, dim=20, ncomp=5, k=12, seed=20 + i)
            rng = np.random.default_rng(i)
            y = rng.standard_normal((6, d))[rng.integers(0, 6, n)] + 0.2 * rng.standard_normal((n, d))
            y = (y * (extent / (y.max(0) - y.min(0)).max())).astype(np.float32)
            p = S.default_params(d=d, format=S.FORMAT_CSR, max_iter=8, alpha=1.0, h=H[d])
            job = S.Job(ctx, p, rp, col, val.astype(np.float32), device_mem=False)
            job.set_y(y, S.LAYOUT_POINT_MAJOR, False)
            jobs.append((job, rp, col, val.astype(np.float32).astype(np.float64), n, d))
        batch = S.Batch(ctx, [j[0] for j in jobs], 1)
        at = lambda job, n, d: job.get_y(np.empty((n, d), np.float32), S.LAYOUT_POINT_MAJOR, False,
                                         0).astype(np.float64)
        u = [np.zeros((j[4], j[5])) for j in jobs]
        g = [np.ones((j[4], j[5])) for j in jobs]
        # how far the momentum may be off; coordinates whose gain is known
        loose, known = [0.0 for _ in jobs], [np.ones((j[4], j[5]), bool) for j in jobs]
        other = 0
        for _ in range(6):
            before = [at(j[0], j[4], j[5]) for j in jobs]
            batch.run(1)
            for i, (job, rp, col, val, n, d) in enumerate(jobs):
                y = before[i] - before[i].mean(0)
                Fr, Z, N, _ = oracle.repulsive_interp(y, H[d])
                assert job.info().error_flags == 0
                dy = oracle.attractive(rp, col, val, y) - Fr
                err = 1e-5 * np.sqrt((dy ** 2).mean())
                step = at(job, n, d) - y
                sure = (np.abs(dy) > err) & ((np.abs(u[i]) > loose[i]) | (u[i] == 0))
                rule = np.sign(dy) != np.sign(u[i])
                new = [np.maximum(np.where(r, g[i] + 0.2, g[i] * 0.8), 0.01) for r in (rule, ~rule)]
                to = [0.5 * u[i] - eta * x * dy for x in new]
                off = [np.abs(step - t) for t in to]
                flip = ~sure & (off[1] < off[0])
                g[i] = np.where(flip, new[1], new[0])
                loose[i] = 0.5 * loose[i] + eta * g[i] * err
                tol = loose[i] + 4 * 2.0 ** -24 * np.abs(y).max()
                assert (np.where(flip, off[1], off[0]) <= tol)[known[i]].all()
                # where the two gains' steps cannot be told apart, the coordinate is left out
                known[i] &= sure | (np.abs(to[0] - to[1]) > 2 * tol)
                u[i] = np.where(flip, to[1], to[0])
                other += int((flip & known[i]).sum())
        assert all(k.mean() > 0.99 for k in known)
        print(f"\n{other} gains decided by rounding")
        batch.close()
        for j in jobs:
            j[0].close()
    finally:
        ctx.close()
