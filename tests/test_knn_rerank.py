"""The automatic kNN search on few points, and its exact re-ranking, against
the SIMT search: the same indices and the same distance bits.

Dimensions at the edges of the re-ranking's runs of 32, and in each of its
copy widths (rows of 4, 2 and 1 floats; 'shift' starts the points off a
16-byte boundary); point counts at the edges of the rule that picks the
search.  'tiny' points have products below the smallest normal number and
'nan' a coordinate that is not a number: such queries must all be redone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,k,kind", [
    (256, 32, 10, "blobs"), (255, 32, 10, "blobs"), (257, 36, 31, "blobs"), (700, 4, 12, "blobs"),
    (700, 30, 33, "blobs"), (700, 34, 64, "blobs"), (700, 31, 97, "blobs"), (700, 33, 128, "blobs"),
    (1024, 2, 3, "blobs"), (1023, 2, 3, "blobs"), (600, 132, 40, "shift"), (600, 66, 15, "shift"),
    (600, 20, 15, "tiny"), (600, 20, 15, "nan"), (1500, 96, 20, "same"),
])
def test_auto_equals_simt_on_few_points(n, dim, k, kind):
    import torch

    import sgtsne_b200 as S
    rng = np.random.default_rng(n + dim + k)
    X = (rng.standard_normal((8, dim)) * 4)[rng.integers(0, 8, n)]
    X = X + rng.standard_normal((n, dim))
    if kind == "tiny":
        X *= 1e-20
    elif kind == "nan":
        X[n // 2, dim // 2] = np.nan
    elif kind == "same":
        X[:] = X[0]
    off = 1 if kind == "shift" else 0
    buf = torch.zeros(n * dim + 4, device="cuda")
    Xd = buf[off:off + n * dim]
    Xd.copy_(torch.from_numpy(np.ascontiguousarray(X, np.float32)).reshape(-1))
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
