"""Batches whose jobs sort dense grids by cell (75,000 points and more, in a
batch of 150,000 and more) beside jobs that scatter, on grids on either side of
what each form and each convolution takes, and the same jobs launched alone
before and after.  Each stretch of two iterations against the same stretch
alone from the same start; bar: the repository's for two iterations in the mix
(1e-5).  The graph is a ring of each point's next neighbours: S2G and G2S do not
depend on it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = {1: 0.5, 2: 0.7, 3: 1.2}


def make(S, ctx, n, d, k=6):
    import torch
    rp = torch.arange(0, (n + 1) * k, k, dtype=torch.int32, device="cuda")
    col = (torch.arange(n, device="cuda")[:, None] + torch.arange(1, k + 1, device="cuda")) % n
    val = torch.full((n * k,), 1.0 / (n * k), device="cuda")
    torch.cuda.synchronize()
    p = S.default_params(d=d, format=S.FORMAT_CSR, max_iter=8, alpha=1.0, h=H[d])
    return S.Job(ctx, p, rp, col.reshape(-1).to(torch.int32), val, device_mem=True)


def state(n, d, extent, seed):
    rng = np.random.default_rng(seed)
    y = rng.uniform(-0.5, 0.5, (n, d)) * extent
    y[: n // 4] *= 0.2
    return y.astype(np.float32)


def get(S, job, n, d):
    return job.get_y(np.empty((n, d), np.float32), S.LAYOUT_POINT_MAJOR, False, 0)


# (points, extent in units of h) of the jobs of one dimension
CASES = [
    (2, [(80000, 12.0), (75000, 46.0), (74999, 12.0), (3000, 30.0), (1500, 140.0)]),
    (2, [(80000, 60.0), (90000, 12.0)]),
    (3, [(80000, 12.0), (76000, 30.0), (2500, 12.0), (2000, 46.0), (1500, 77.0),
         (1500, 90.0)]),
    (1, [(100000, 12.0), (80000, 300.0), (2000, 40.0)]),
]


@pytest.mark.parametrize("d,jobs", CASES)
def test_in_a_batch_as_alone(d, jobs):
    import sgtsne_b200 as S
    rel = lambda a, b: np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b)
    ctx = S.Context(0)
    try:
        made = [make(S, ctx, n, d) for n, _ in jobs]
        alone = [make(S, ctx, n, d) for n, _ in jobs]
        batch = S.Batch(ctx, made, 2)
        few = S.Batch(ctx, made[:1], 1)
        for i, ((n, e), a, b) in enumerate(zip(jobs, made, alone)):
            y = state(n, d, e * H[d], 10 * d + i)
            a.set_y(y, S.LAYOUT_POINT_MAJOR, False)
            b.set_y(y, S.LAYOUT_POINT_MAJOR, False)
        # together, alone again, in a batch too small for the batch's rules, together
        for step in ("batch", "alone", "few", "batch"):
            if step == "batch":
                batch.run(2)
            elif step == "few":
                few.run(2)
            for i, ((n, _), a, b) in enumerate(zip(jobs, made, alone)):
                if step == "few" and i > 0:
                    continue
                if step == "alone":
                    a.run(2)
                b.run(2)
                ya, yb = get(S, a, n, d), get(S, b, n, d)
                assert rel(ya, yb) <= 1e-5, (step, i)
                assert a.info().error_flags == 0 and b.info().error_flags == 0
                assert a.info().grid_points == b.info().grid_points
        batch.close()
        few.close()
        for j in made + alone:
            j.close()
    finally:
        ctx.close()
