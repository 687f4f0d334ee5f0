"""Which results share the pinned buffer, and which copies they take (nsem_copy.h),
on plain memory with a recording copy: no GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r"""
#include <cstring>
#include "nsem_copy.h"
/* results i = 0..n-1: values [src[i], src[i] + len[i]) of dev to dst + 100 i;
 * pageable[i]; room of the buffer in bytes; log: (destination, source, values)
 * of every copy, the destination as its offset in the buffer or -1 - i.
 * Returns the copies made, staged in *staged. */
extern "C" int run(const double* dev, const int* src, const int* len, const int* pageable, int n,
                   double* dst, double* buffer, int room, int* log, int* staged) {
    NsemHostCopy c[8];
    for (int i = 0; i < n; i++) c[i] = {dst + 100 * i, dev + src[i], (size_t)len[i]};
    *staged = nsem_stage_results(c, n, (size_t)room,
                                 [&](const double* p) { return pageable[(p - dst) / 100] != 0; });
    int k = 0;
    nsem_copy_results(c, n, *staged ? buffer : nullptr, [&](double* d, const double* s, size_t m) {
        log[3 * k] = *staged ? (int)(d - buffer) : -1 - (int)((d - dst) / 100);
        log[3 * k + 1] = (int)(s - dev);
        log[3 * k + 2] = (int)m;
        k++;
        std::memcpy(d, s, m * sizeof(double));
        return 0;
    });
    return k;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("copy")
    (d / "h.cpp").write_text(HARNESS)
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "nebulasem_gb300", "csrc"), str(d / "h.cpp"), "-o",
                    str(d / "libh.so")], check=True)
    return ctypes.CDLL(str(d / "libh.so"))


def _run(lib, src, length, pageable, room):
    n = len(src)
    ints = lambda v: (ctypes.c_int * len(v))(*v)
    dev = (ctypes.c_double * 1000)(*range(1000))
    dst, buf = (ctypes.c_double * 800)(), (ctypes.c_double * 1000)()
    log, staged = ints([0] * 24), ctypes.c_int()
    k = lib.run(dev, ints(src), ints(length), ints(pageable), n, dst, buf, room, log, ctypes.byref(staged))
    return bool(staged.value), [tuple(log[3 * i:3 * i + 3]) for i in range(k)]


@pytest.mark.parametrize("pageable,staged", [((1, 1, 1), True), ((0, 1, 1), False), ((1, 0, 1), False),
                                             ((1, 1, 0), False)])
def test_every_destination_is_looked_at(lib, pageable, staged):
    got, copies = _run(lib, (0, 50, 200), (10, 10, 30), pageable, 400)
    assert got is staged
    assert copies == ([(0, 0, 10), (10, 50, 10), (20, 200, 30)] if staged
                      else [(-1, 0, 10), (-2, 50, 10), (-3, 200, 30)])


@pytest.mark.parametrize("room,staged", [(400, True), (399, False), (0, False)])
def test_room_of_the_buffer(lib, room, staged):
    assert _run(lib, (0, 50, 200), (10, 10, 30), (1, 1, 1), room)[0] is staged


def test_a_single_result_is_copied_directly(lib):
    assert _run(lib, (7,), (10,), (1,), 400) == (False, [(-1, 7, 10)])
