"""Staged results are joined into one copy where the caller states that they
share an allocation, never because their addresses happen to follow each other
(nsem_copy.h); no GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include "nsem_copy.h"
/* four results of 10 values, neighbours in dev; the values of each copy in sizes */
extern "C" int run(const double* dev, const int* joins, double* dst, double* buffer, int* sizes) {
    NsemHostCopy c[4];
    for (int i = 0; i < 4; i++) c[i] = {dst + 10 * i, dev + 10 * i, 10, joins[i] != 0};
    int k = 0;
    nsem_copy_results(c, 4, buffer, [&](double*, const double*, size_t m) {
        sizes[k++] = (int)m;
        return 0;
    });
    return k;
}
"""


@pytest.mark.parametrize("joins,staged,want", [((0, 0, 0, 0), 1, [10, 10, 10, 10]), ((0, 1, 1, 1), 1, [40]),
                                               ((0, 1, 0, 1), 1, [20, 20]), ((0, 1, 1, 1), 0, [10, 10, 10, 10])])
def test_joined_only_where_stated(tmp_path, joins, staged, want):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "nebulasem_gb300", "csrc"), str(tmp_path / "h.cpp"), "-o",
                    str(tmp_path / "libh.so")], check=True)
    lib = ctypes.CDLL(str(tmp_path / "libh.so"))
    dev, dst, buf = ((ctypes.c_double * 40)() for _ in range(3))
    sizes = (ctypes.c_int * 4)()
    k = lib.run(dev, (ctypes.c_int * 4)(*joins), dst, buf if staged else None, sizes)
    assert list(sizes[:k]) == want
