"""Data whose squared norms FP32 cannot sum (one large coordinate, hundreds of
small ones), and data far from the origin: the automatic kNN search against the
SIMT search, the same indices and the same distance bits.

'sums' is the case of test_knn_bound_model.py in one term (BF16 numbers),
'sums3' in three; in 'offset' the norms are 1e8 times the distances' spread.
"""
import numpy as np
import pytest

import test_knn_bound_model as model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dim,k", [("sums", 784, 15), ("sums3", 784, 15), ("sums", 1100, 20),
                                        ("offset", 16, 10), ("offset", 300, 40)])
def test_auto_equals_simt_where_norms_are_large(kind, dim, k):
    both_searches(model.points(kind, dim, np.random.default_rng(799)), k)


@pytest.mark.parametrize("n,dim,k", [(1623, 2, 1), (1624, 2, 1), (1474, 31, 2), (1174, 3, 4),
                                     (1024, 32, 1), (1024, 4, 5)])
def test_auto_equals_simt_at_its_least_points(n, dim, k):
    rng = np.random.default_rng(n + dim)
    X = (rng.standard_normal((8, dim)) * 4)[rng.integers(0, 8, n)] + rng.standard_normal((n, dim))
    both_searches(np.ascontiguousarray(X, np.float32), k)


def both_searches(X, k):
    import torch

    import sgtsne_b200 as S
    n, dim = X.shape
    Xd = torch.from_numpy(X).cuda()
    ctx = S.Context(0)
    out = []
    try:
        for method in (S.KNN_SIMT, S.KNN_AUTO):
            idx = torch.full((n * k,), -7, dtype=torch.int32, device="cuda")
            d2 = torch.full((n * k,), -7.0, dtype=torch.float32, device="cuda")
            torch.cuda.synchronize()
            ctx.knn(n, dim, Xd, k, idx, d2, method=method)
            out.append((idx.cpu().numpy(), d2.cpu().numpy().view(np.uint32)))
    finally:
        ctx.close()
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
