"""The automatic kNN search (tensor-core filter from 4096 points on) against
the SIMT search: the same indices and the same distance bits, for widths and
list lengths on either side of the filter's limits.

'ints' are 8-bit values, exact in BF16 (one product term); 'blobs' are not
(three terms).  'grid' ties everywhere.  'runs' puts the points of small
clusters next to each other, so that all neighbours of a query fall in one
half of a candidate tile.  64 and 65 dimensions: resident and streamed query
images; 33, 96, 97 and 128 neighbours: the edges of the list sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k,kind", [
    (5000, 784, 90, "ints"), (4096, 65, 33, "blobs"), (5003, 64, 96, "blobs"),
    (4353, 130, 97, "blobs"), (4100, 17, 128, "ints"), (4500, 3, 33, "grid"),
    (4608, 40, 30, "runs"), (5000, 257, 1, "runs"), (4099, 1, 5, "blobs"),
])
def test_auto_equals_simt(n, dim, k, kind):
    import torch

    import sgtsne_b200 as S
    rng = np.random.default_rng(n + dim + k)
    if kind == "ints":
        X = rng.integers(0, 256, (n, dim)) * (rng.random((n, dim)) < 0.3)
    elif kind == "grid":
        X = rng.integers(0, 12, (n, dim))
    elif kind == "runs":
        X = np.repeat(rng.standard_normal((n // 48 + 1, dim)) * 8, 48, 0)[:n]
        X = X + rng.standard_normal((n, dim))
    else:
        X = (rng.standard_normal((8, dim)) * 4)[rng.integers(0, 8, n)]
        X = X + rng.standard_normal((n, dim))
    Xd = torch.from_numpy(np.ascontiguousarray(X, np.float32)).cuda()
    ctx = S.Context(0)
    out = []
    try:
        for method in (S.KNN_SIMT, S.KNN_AUTO):
            idx = torch.full((n * k,), -7, dtype=torch.int32, device="cuda")
            d2 = torch.full((n * k,), -7.0, dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            redo = ctx.knn(n, dim, Xd, k, idx, d2, method=method)
            out.append((idx.cpu().numpy(), d2.cpu().numpy().view(np.uint32)))
    finally:
        ctx.close()
    print(f"\nknn n={n} dim={dim} k={k} {kind}: {redo} queries redone")
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
