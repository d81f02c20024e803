"""The rules by which a grid's size picks the form of the repulsion and the
points' number that of the kNN search (gpu-sg-sne_b200/csrc/sgt_grid_rules.h and
sgt_knn_rules.h, compiled from those files) against
measurements: where one form took a tenth longer than the other on a B200, the
rule must not pick it.  Times are us per iteration of CSR jobs with k = 30.
"""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "gpu-sg-sne_b200", "csrc")

# (d, points, points per axis, sorted by cell, scattered)
CELL = [
    (1, 50000, 16, 35.3, 31.0), (1, 50000, 64, 37.4, 27.6), (1, 100000, 16, 42.8, 49.2),
    (1, 100000, 125, 43.3, 40.4), (1, 150000, 16, 53.5, 65.8), (1, 200000, 16, 67.3, 85.8),
    (1, 290000, 16, 83.7, 111.4), (1, 290000, 500, 86.5, 80.4),
    (2, 50000, 16, 48.4, 39.2), (2, 75000, 25, 53.0, 45.6), (2, 100000, 40, 63.7, 57.6),
    (2, 200000, 16, 79.6, 95.2), (2, 200000, 40, 80.6, 92.7), (2, 200000, 66, 95.0, 89.1),
    (2, 290000, 16, 106.5, 126.2), (2, 290000, 56, 103.7, 121.9),
    (3, 50000, 16, 102.9, 71.2), (3, 75000, 16, 104.7, 88.8), (3, 100000, 16, 111.4, 103.2),
    (3, 200000, 16, 137.5, 163.6), (3, 290000, 16, 167.2, 217.5),
]


# 3-D: (nonzeros of P in millions, points per axis, FFT length, plain transforms,
# FFT passes)
CONV = [
    (0.1, 25, 64, 46, 54), (0.1, 28, 64, 62, 55), (0.1, 39, 96, 86, 104), (0.1, 48, 96, 152, 113),
    (0.1, 63, 128, 282, 184), (0.1, 72, 192, 489, 640), (1.5, 20, 64, 65, 76),
    (1.5, 32, 64, 99, 81), (1.5, 40, 96, 121, 128), (1.5, 48, 96, 173, 135),
    (1.5, 56, 128, 238, 192), (1.5, 64, 128, 348, 201), (1.5, 66, 192, 438, 623),
    (5, 32, 64, 143, 125), (5, 40, 96, 178, 172), (5, 48, 96, 248, 180), (5, 50, 128, 256, 226),
    (5, 56, 128, 309, 235), (5, 66, 192, 517, 644), (5, 78, 192, 760, 715),
    (15, 40, 96, 287, 300), (15, 48, 96, 358, 294), (15, 64, 128, 593, 384),
    (15, 66, 192, 713, 795), (15, 78, 192, 1007, 872),
]


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src = d / "r.cpp"
    src.write_text('#include "sgt_grid_rules.h"\n#include "sgt_knn_rules.h"\n'
                   'extern "C" int knn_min_n(int dim, int k) { return sgt_knn_min_n(dim, k); }\n'
                   'extern "C" int cell(int d, long n, long ncell) {\n'
                   '  return n >= sgt_cell_min_n(d) && sgt_cell_mode(n, ncell, SGT_CELL_DENSE);\n'
                   '}\n'
                   'extern "C" int plain(int d, int N, int M, int work) {\n'
                   '  return sgt_plain_conv(d, N, M, SGT_SPEC_MAX(d),\n'
                   '                        work ? SGT_CONV_WORK_LONG : SGT_CONV_WORK);\n'
                   '}\n'
                   'extern "C" int copies(int d, long n, int N) {\n'
                   '  const long nodes = d == 2 ? (long)N * N : (long)N * N * N;\n'
                   '  return sgt_copies((n << (2 * d)) / nodes, nodes, d == 2 ? 1l << 18 : 1l << 21,\n'
                   '                    sgt_copy_adds(d), SGT_COPIES);\n'
                   '}\n'
                   'extern "C" int fft(int d, int nmax) {\n'
                   '  return sgt_needs_fft(d, nmax, nmax < SGT_SPEC_MAX(d) ? nmax : SGT_SPEC_MAX(d));\n'
                   '}\n')
    so = d / "r.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.cell.argtypes = [ctypes.c_int, ctypes.c_long, ctypes.c_long]
    lib.copies.argtypes = [ctypes.c_int, ctypes.c_long, ctypes.c_int]
    return lib


@pytest.mark.parametrize("d,n,N,by_cell,scattered", CELL)
def test_cell_mode(rules, d, n, N, by_cell, scattered):
    picked = bool(rules.cell(d, n, (N - 3) ** d))
    assert (by_cell if picked else scattered) < 1.1 * min(by_cell, scattered)


@pytest.mark.parametrize("nnz,N,M,plain,fft", CONV)
def test_convolution_of_3d_grids(rules, nnz, N, M, plain, fft):
    picked = bool(rules.plain(3, N, M, int(nnz >= 3)))
    # (28 points of a light job: 62 / 55, within two of 25's 46 / 54)
    assert (plain if picked else fft) < 1.13 * min(plain, fft)


def test_a_job_whose_grids_can_take_the_passes_has_them(rules):
    sizes = [8, 9, 10, 11, 12, 13, 14, 15, 16, 20, 25, 26, 28, 32, 33, 35, 36, 39, 40, 42, 44, 45,
             48, 49, 50, 52, 54, 55, 56, 60, 63, 64, 65, 66, 70, 72, 75, 77, 78, 80, 84, 88, 128]
    lengths = [32, 64, 96, 128, 192, 256]
    for d in (2, 3):
        for nmax in sizes:
            takes = any(not rules.plain(d, N, next(m for m in lengths if m >= 2 * N - 1), long)
                        for N in sizes if N <= nmax for long in (0, 1))
            assert rules.fft(d, nmax) >= takes


# (d, points, points per axis, {adds per copy: us per iteration})
@pytest.mark.parametrize("d,n,N,us", [
    (3, 100000, 25, {16: 131, 32: 122, 64: 121, 128: 129}),
    (3, 299000, 40, {16: 328, 32: 287, 64: 294, 128: 305}),
    (3, 299000, 48, {16: 321, 32: 294, 64: 287, 128: 302}),
    (3, 299000, 64, {16: 425, 32: 384, 64: 386, 128: 414}),
    (2, 100000, 40, {16: 56, 32: 55, 64: 60, 128: 62}),
    (2, 299000, 200, {16: 137, 32: 136, 64: 148, 128: 148}),
])
def test_grid_copies(rules, d, n, N, us):
    adds, fit = (n << (2 * d)) // N ** d, (1 << (18 if d == 2 else 21)) // N ** d

    def copies(per):
        c = 1
        while c < 32 and per * c < adds and 2 * c <= fit:
            c *= 2
        return c
    picked = [t for per, t in us.items() if copies(per) == rules.copies(d, n, N)]
    assert picked and min(picked) <= 1.06 * min(us.values())


# (dim, k, points, us of the filter, us of the SIMT search)
@pytest.mark.parametrize("dim,k,n,tensor,simt", [
    (2, 1, 1024, 276, 192), (2, 1, 1500, 288, 273), (2, 1, 2048, 334, 360), (2, 4, 1024, 274, 262),
    (2, 4, 1500, 297, 347), (2, 9, 1024, 273, 430), (2, 10, 256, 175, 183), (10, 1, 1024, 285, 216),
    (10, 1, 2048, 346, 407), (10, 4, 1500, 308, 394), (10, 15, 256, 178, 281),
    (50, 1, 1024, 309, 337), (50, 4, 1024, 311, 438), (50, 10, 256, 202, 237),
    (784, 10, 256, 483, 959),
])
def test_choice_of_the_knn_search(rules, dim, k, n, tensor, simt):
    assert (tensor if n >= rules.knn_min_n(dim, k) else simt) <= 1.05 * min(tensor, simt)
