"""Scatter mode and cell mode of the repulsion, and the two convolutions, at
the sizes where one takes over from the other, against the FP64 oracle on the
same grid.

The convolution in Fourier space along x with direct row sums takes grids up
to 128 points per axis in 2-D and 40 in 3-D (the size table's neighbours are
126 and 130, 40 and 42); 1-D grids up to 512 are summed directly.  500 points
need one copy of the grid, 40,000 clustered ones up to 32.  300,000 points on
13^2 or 13^3 cells are the fewest that are sorted by cell.  Bars: those of the
parity table (charge grid 1e-5, potentials 1e-4, forces 3e-4, Z 5e-4), which
hold FP32 sums of 4^d-point stencils on any of these grids.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


@pytest.mark.parametrize("d,n,ng", [
    (1, 500, 6), (1, 40000, 510),
    (2, 500, 6), (2, 500, 124), (2, 40000, 14), (2, 40000, 62), (2, 40001, 124), (2, 40000, 127),
    (3, 500, 6), (3, 40001, 18), (3, 40000, 38), (3, 3000, 40),
    (2, 299999, 14), (2, 300000, 14), (3, 300000, 14),
])
def test_modes_against_oracle(d, n, ng):
    import torch

    import sgtsne_b200 as S
    from oracle import oracle as O
    ctx = S.Context(0)
    try:
        rng = np.random.default_rng(1000 * d + ng)
        h = {1: 0.5, 2: 0.7, 3: 1.2}[d]
        c = rng.standard_normal((6, d)) * 3
        Y = (c[rng.integers(0, 6, n)] + rng.standard_normal((n, d)) * 0.4).astype(np.float32)
        f = torch.empty(n * d, dtype=torch.float32, device="cuda")
        Yd = torch.from_numpy(np.ascontiguousarray(Y)).cuda()
        torch.cuda.synchronize()
        for _ in range(2):  # the second call finds the copies the first has used
            Z, N, he = ctx.repulsive(n, d, h, ng, Yd, S.LAYOUT_POINT_MAJOR, f)
        assert N == S.best_grid_size(ng) + 2
        V, Phi = ctx.last_grids(d, N)
    finally:
        ctx.close()
    _, sc, sh, N2, mx = O.bins_f32(Y, h, S.best_grid_size(ng))
    assert N2 == N
    q = np.concatenate([np.ones((n, 1)), sh.astype(np.float64) - 0.5 * float(mx)], 1)
    assert rel(V, O.s2g(sc.astype(np.float64), q, N)) <= 1e-5
    assert rel(Phi, O.g2g(V.astype(np.float64), float(he), 0)) <= 1e-4
    Fo, Zo, No, _ = O.repulsive_interp(Y.astype(np.float64), h, n1_force=N - 2)
    assert No == N
    assert abs(Z - Zo) <= 5e-4 * abs(Zo)
    assert rel(f.cpu().numpy().reshape(n, d), Fo) <= 3e-4
