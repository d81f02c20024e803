"""The rules by which a grid's size picks the form of the repulsion
(gpu-sg-sne_b200/csrc/sgt_grid_rules.h, compiled from that file) against
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


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src = d / "r.cpp"
    src.write_text('#include "sgt_grid_rules.h"\n'
                   'extern "C" int cell(int d, long n, long ncell) {\n'
                   '  return n >= sgt_cell_min_n(d) && sgt_cell_mode(n, ncell, SGT_CELL_DENSE);\n'
                   '}\n')
    so = d / "r.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, str(src), "-o",
                    str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.cell.argtypes = [ctypes.c_int, ctypes.c_long, ctypes.c_long]
    return lib


@pytest.mark.parametrize("d,n,N,by_cell,scattered", CELL)
def test_cell_mode(rules, d, n, N, by_cell, scattered):
    picked = bool(rules.cell(d, n, (N - 3) ** d))
    assert (by_cell if picked else scattered) < 1.1 * min(by_cell, scattered)
