"""The sort by cell inside runs: a captured job whose grid passes from the sort
to the scatter and back while it runs, and a row-split embedding that sorts
because the whole embedding is large.

200,000 points are the fewest a 2-D job sorts; on 56 points per axis a cell holds
71 of them, on 60 (the next size) 62, below the 64 of the rule.  The coordinates
start just inside 54 steps of h, spread by their repulsion past them, and are
set back.  The graph is a ring of each point's next three neighbours.

Bar of the runs: six iterations against the FP64 oracle, 1e-5 (FP32 coordinates
and sums; gains that rounding decides differently move single points).  The
shard runs the same kernels as the job from statistics summed in another order:
1e-5 after three iterations.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_PTS = 200000


def ring(n, k=3):
    rp = np.arange(0, (2 * k) * n + 1, 2 * k, dtype=np.int32)
    off = np.r_[-k:0, 1:k + 1]
    col = np.sort((np.arange(n)[:, None] + off) % n, 1).reshape(-1).astype(np.int32)
    return rp, col, np.full(2 * k * n, 1.0 / (2 * k * n), np.float32)


def state(steps, seed):
    """Uniform points exactly `steps` steps of h = 0.7 wide."""
    y = np.random.default_rng(seed).uniform(0.0, 1.0, (N_PTS, 2))
    y = (y - y.min(0)) / (y.max(0) - y.min(0)) - 0.5
    return (y * (0.7 * steps)).astype(np.float32)


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def test_a_run_through_both_modes(oracle):
    import sgtsne_b200 as S
    rp, col, val = ring(N_PTS)
    p = S.default_params(d=2, format=S.FORMAT_CSR, max_iter=600, alpha=1.0, h=0.7)
    ctx = S.Context(0)
    try:
        job = S.Job(ctx, p, rp, col, val, device_mem=False)
        for y0, grids in ((state(53.99999, 1), {56, 60}), (state(13.0, 2), {16}),
                          (state(70.0, 3), {77}), (state(53.99999, 1), {56, 60})):
            job.set_y(y0, S.LAYOUT_POINT_MAJOR, False)
            seen = set()
            for _ in range(6):
                seen.add(job.info().grid_points)
                job.run(1)
            y = job.get_y(np.empty((N_PTS, 2), np.float32), S.LAYOUT_POINT_MAJOR, False, 1)
            assert job.info().error_flags == 0
            want = oracle.kl_minimization(rp, col, val.astype(np.float64), y0.astype(np.float64), 6,
                                          alpha=1.0, h=0.7)
            print("\ngrids", sorted(seen), "error", rel(y, want - want.mean(0)))
            assert rel(y, want - want.mean(0)) <= 1e-5
            if len(grids) > 1:
                assert seen == grids
        job.close()
    finally:
        ctx.close()


def test_a_shard_sorts_as_the_whole_embedding_would():
    import torch
    import torch.distributed as dist
    from test_sharded import _free_port

    import sgtsne_b200 as S
    from sgtsne_b200.sharded import EngineShard, ShardedEmbedding
    rp, col, val = ring(N_PTS)
    p = S.default_params(d=2, format=S.FORMAT_CSR, max_iter=8, alpha=1.0, h=0.7, max_grid=128)
    torch.cuda.set_device(0)
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    ctx = S.Context(0)
    ctx.set_stream(stream.cuda_stream)
    dist.init_process_group("nccl", init_method=f"tcp://127.0.0.1:{_free_port()}", rank=0,
                            world_size=1)
    try:
        for steps in (20.0, 70.0):
            y0 = state(steps, 4)
            sh = EngineShard(ctx, p, N_PTS, 0, 1, rp, col, val, "cuda:0")
            sh.set_y(y0)
            ShardedEmbedding(sh).run(3)
            ys = sh.get_y()
            assert sh.info().error_flags == 0
            sh.close()
            job = S.Job(ctx, p, rp, col, val, device_mem=False)
            job.set_y(y0, S.LAYOUT_POINT_MAJOR, False)
            job.run(3)
            yj = job.get_y(np.empty((N_PTS, 2), np.float32), S.LAYOUT_POINT_MAJOR, False, 1)
            job.close()
            assert rel(ys.astype(np.float64), yj) <= 1e-5
    finally:
        dist.destroy_process_group()
        torch.cuda.set_stream(torch.cuda.default_stream())
        ctx.close()
