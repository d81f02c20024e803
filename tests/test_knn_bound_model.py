"""A CPU model of the arithmetic of the tensor-core kNN filter (k_knn_tc in
gpu-sg-sne_b200/csrc/sgt_knn.cu), with the bounds of sgt_knn_rules.h compiled
from that file.

Keys q.c - |c|^2/2 from BF16 parts, in one term (points that are BF16 numbers)
or three; MMAs of 16 dimensions in the kernel's order, each cutting its 16
products and the accumulator at 2^-25 of the largest one's power of two and its
sum to FP32, towards zero; norms summed in FP64.  The L best keys are kept, those within the
bound of the k-th key re-ranked with the SIMT search's FP32 sums, and a query
is settled when everything dropped is farther than the k-th distance.

1. No key is further off than the bound.
2. Every settled query has the SIMT search's neighbours and distances.
3. The bound is of use: ordinary data settle.
4. The case of large norms that FP32 cannot sum is one: with FP32 norms and
   2^-21 a step, the same model settles queries wrongly.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpu-sg-sne_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src = d / "r.cpp"
    src.write_text('#include "sgt_knn_rules.h"\n'
                   'extern "C" float eps(int dim, int exact) { return sgt_knn_eps(dim, exact); }\n'
                   'extern "C" float gam(int dim) { return sgt_knn_gamma(dim); }\n')
    so = d / "r.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.eps.restype = lib.gam.restype = ctypes.c_float
    return lib


def bf16(x):
    """Round to nearest even to 8 significant bits (finite values)."""
    b = np.ascontiguousarray(x, np.float32).view(np.uint32)
    r = (b + np.uint32(0x7FFF) + ((b >> np.uint32(16)) & np.uint32(1))) & np.uint32(0xFFFF0000)
    return r.astype(np.uint32).view(np.float32)


def trunc32(x):
    """FP64 to FP32 towards zero."""
    f = x.astype(np.float32)
    over = np.abs(f.astype(np.float64)) > np.abs(x)
    return np.where(over, np.nextafter(f, np.float32(0)), f).astype(np.float64)


def mma(acc, a, b):
    """acc[q, c] + sum over 16 dimensions of a[q] b[c], as stated above."""
    p = a[:, None, :].astype(np.float64) * b[None].astype(np.float64)
    p = np.concatenate([p, acc[..., None]], -1)
    e = np.frexp(np.abs(p).max(-1))[1]  # the largest's power of two is 2^(e - 1)
    unit = np.ldexp(1.0, e - 26)[..., None]
    return trunc32((np.trunc(p / unit) * unit).sum(-1))


def norms64(X):
    return (X.astype(np.float64) ** 2).sum(1).astype(np.float32)


def norms32(X):
    s = np.zeros(len(X), np.float32)
    for k in range(X.shape[1]):  # multiply-adds rounded once
        s = (s.astype(np.float64) + X[:, k].astype(np.float64) ** 2).astype(np.float32)
    return s


def keys(X, Q, nrm, exact):
    """Key of every candidate for the query rows Q."""
    n, dim = X.shape
    U = (dim + 3 + 15) // 16 * 2
    hi, lo = bf16(X), bf16(X - bf16(X))
    A, AL = np.zeros((len(Q), 8 * U), np.float32), np.zeros((len(Q), 8 * U), np.float32)
    B, BL = np.zeros((n, 8 * U), np.float32), np.zeros((n, 8 * U), np.float32)
    A[:, :dim], AL[:, :dim], B[:, :dim], BL[:, :dim] = hi[Q], lo[Q], hi, lo
    A[:, dim:dim + 3] = 1.0
    half = np.float32(-0.5) * nrm
    for c in range(3):
        B[:, dim + c] = bf16(half)
        half = half - bf16(half)
    ku = 4 if U <= 8 else 8
    acc = np.zeros((len(Q), n))
    for c0 in range(0, U, ku):
        for a, b in ((A, B), (A, BL), (AL, B))[:1 if exact else 3]:
            for u in range(c0, min(c0 + ku, U), 2):
                acc = mma(acc, a[:, 8 * u:8 * u + 16], b[:, 8 * u:8 * u + 16])
    return acc


def simt(X, q, c):
    """FP32 sums of squared differences in dimension order."""
    s = np.zeros(len(c), np.float32)
    df = (X[q] - X[c]).astype(np.float32).astype(np.float64)
    for k in range(X.shape[1]):
        s = (s.astype(np.float64) + df[:, k] ** 2).astype(np.float32)
    return s


def nearest(d, c, k):
    o = np.lexsort((c, d))[:k]
    return c[o], d[o]


def search(X, Q, k, eps, gamma, norms):
    """(settled, indices, distances) per query and the keys' largest error over
    |q|^2 + max |c|^2."""
    n, dim = X.shape
    L = 64 if k <= 32 else (128 if k <= 96 else 192)
    exact = bool((bf16(X) == X).all())
    nrm = norms(X)
    K = keys(X, Q, nrm, exact)
    X64 = X.astype(np.float64)
    true = (X64[Q] ** 2).sum(1)[:, None] - ((X64[Q][:, None] - X64[None]) ** 2).sum(-1)
    scale = nrm[Q].astype(np.float64) + float(nrm.max())
    err = (np.abs(2 * K - true) / scale[:, None]).max()
    out = []
    for i, q in enumerate(Q):
        c = np.delete(np.arange(n), q)
        ky = K[i, c]
        o = np.argsort(-ky, kind="stable")
        tail = ky[o[L]] if len(o) > L else -np.inf
        bound = float(np.float32(eps) * np.float32(scale[i]))
        qn, kth = float(nrm[q]), ky[o[k - 1]]
        far = max(qn - 2 * kth + bound, 0.0)
        keep = o[:L][ky[o[:L]] >= kth - (bound + 1.1 * gamma * far)]
        idx, d = nearest(simt(X, q, c[keep]), c[keep], k)
        near = qn - 2 * tail - bound
        out.append((tail == -np.inf or near - 1.1 * gamma * near > d[-1], idx, d))
    return out, err


def points(kind, dim, rng):
    if kind == "blobs":
        X = (rng.standard_normal((8, dim)) * 5)[rng.integers(0, 8, 700)]
        X = X + rng.standard_normal((700, dim))
    elif kind == "ints":
        X = rng.integers(0, 256, (5, dim))[rng.integers(0, 5, 500)] * (rng.random((500, dim)) < 0.3)
    elif kind == "offset":
        X = 1000.0 + 0.1 * rng.standard_normal((400, dim))
    else:  # 'sums': FP32 sums of the squares round up by 2 at each of 700 nonzeros
        v = 1.421875 if kind == "sums" else 1.421875 * (1 + 2.0 ** -11)
        X = np.zeros((421, dim))
        X[0, 1:701] = v
        for i in range(1, 21):
            X[i] = X[0]
            X[i, rng.choice(np.arange(1, 701), 30, False)] = 0
            X[i, rng.choice(np.arange(701, dim), 30, False)] = v
        for i in range(21, 421):
            X[i, rng.choice(np.arange(1, 701), 350, False)] = v
        X[:, 0] = 5824.0
    return np.ascontiguousarray(X, np.float32)


@pytest.mark.parametrize("kind,dim,k,least", [
    ("blobs", 50, 30, 0.95), ("blobs", 3, 10, 0.95), ("blobs", 130, 97, 0.9), ("ints", 60, 30, 0.9),
    ("ints", 784, 90, 0.9), ("blobs", 63, 30, 0.95), ("blobs", 784, 90, 0.0), ("offset", 16, 10, 0.0), ("sums", 784, 15, 0.0), ("sums3", 784, 15, 0.0),
])
def test_settled_queries_are_right(rules, kind, dim, k, least):
    rng = np.random.default_rng(dim + k)
    X = points(kind, dim, rng)
    Q = np.r_[0:21] if kind.startswith("sums") else rng.choice(len(X), 24, False)
    exact = bool((bf16(X) == X).all())
    assert exact == (kind in ("ints", "sums"))
    eps, gamma = rules.eps(dim, int(exact)), rules.gam(dim)
    out, err = search(X, Q, k, eps, gamma, norms64)
    print(f"\n{kind} {dim}-D: error {err:.2e} of {eps:.2e}, settled "
          f"{np.mean([o[0] for o in out]):.2f}")
    assert err <= eps
    for q, (ok, idx, d) in zip(Q, out):
        if ok:
            c = np.delete(np.arange(len(X)), q)
            ti, td = nearest(simt(X, q, c), c, k)
            assert np.array_equal(idx, ti) and np.array_equal(d, td)
    assert np.mean([o[0] for o in out]) >= least


def test_fp32_norms_would_settle_wrongly():
    X = points("sums", 784, np.random.default_rng(799))
    out, _ = search(X, np.r_[0:21], 15, 51 * 4.8e-7, 0.0, norms32)
    c = np.arange(1, len(X))
    right = nearest(simt(X, 0, c), c, 15)[0]
    assert out[0][0] and not np.array_equal(out[0][1], right)
