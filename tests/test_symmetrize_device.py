"""Device symmetrisation against the host's: the same pattern and the same
bits, at the edge between 32-bit and 64-bit keys, with empty rows, a hub,
repeated columns in a row, unsorted columns and entries on the diagonal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (2, 3), (3, 2), (257, 4), (5000, 30), (65536, 3),
                                 (65537, 3), (200000, 2)])
def test_device_equals_host(n, k):
    import torch

    import sgtsne_b200 as S
    rng = np.random.default_rng(n)
    deg = rng.integers(0, 2 * k + 1, n)
    deg[n // 2] = 5 * k  # a hub row
    deg[n // 3:n // 3 + n // 10] = 0  # and a stretch of empty ones
    rp = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    nnz = int(rp[-1])
    if nnz == 0:
        rp[-1] = nnz = 1
    col = rng.integers(0, n, nnz).astype(np.int32)
    col[rng.random(nnz) < 0.1] = n - 1  # a hub column
    val = rng.standard_normal(nnz).astype(np.float32)
    want = S.symmetrize(rp, col, val, 1.0 / (2 * n))
    ctx = S.Context(0)
    try:
        d = [torch.from_numpy(a).cuda() for a in (rp, col, val)]
        orp = torch.empty(n + 1, dtype=torch.int32, device="cuda")
        oc = torch.empty(2 * nnz, dtype=torch.int32, device="cuda")
        ov = torch.empty(2 * nnz, device="cuda")
        torch.cuda.synchronize()
        m = ctx.symmetrize(n, nnz, *d, 1.0 / (2 * n), orp, oc, ov)
    finally:
        ctx.close()
    assert m == len(want[1])
    assert np.array_equal(orp.cpu().numpy(), want[0])
    assert np.array_equal(oc[:m].cpu().numpy(), want[1])
    assert np.array_equal(ov[:m].cpu().numpy().view(np.uint32),
                          np.asarray(want[2], np.float32).view(np.uint32))
