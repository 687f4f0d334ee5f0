"""The integer division, square root, products and power as the device computes
them, against the hardware's operations and the accurate power: the same bits."""
import ctypes
import math
import os
import subprocess

import pytest

from nebulasem_gb300 import build as nb

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
KINDS = ("div", "sqrt", "mul", "signed", "pow", "undecided")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("intfp") / "libintfp.so")
    subprocess.run([nb.nvcc(), *nb.COMMON, *nb.EXACT, "-shared", os.path.join(HERE, "intfp_device.cu"), "-o", so],
                   check=True)
    return ctypes.CDLL(so)


def _run(lib, n=0, seed=0, y=1.4, values=()):
    out = (ctypes.c_ulonglong * len(KINDS))()
    v = (ctypes.c_double * len(values))(*values) if values else None
    e = lib.run(ctypes.c_int64(n), ctypes.c_uint64(seed), ctypes.c_double(y), v, len(values), out)
    assert e == 0
    return dict(zip(KINDS, out))


@pytest.mark.parametrize("y", [1004.5 / 717.5, 2.0 ** -11, 3.7, 7.9])
def test_operations_equal_hardware(lib, y):
    n = 8_000_000
    got = _run(lib, n, 17, y)
    undecided = got.pop("undecided")
    assert got == {k: 0 for k in KINDS[:5]}
    # the rounding test's width: 2 (floor(y) + 2) 2^26 of 2^43 remainders
    assert undecided < 20 + 2 * n * 2 * (int(y) + 2) * 2.0 ** -17


def test_special_operands(lib):
    vals = [0.0, -0.0, 1.0, -1.0, 5e-324, 1e-310, 2.2250738585072014e-308, 1e308, math.inf, -math.inf,
            math.nan, 1e-300, 1e300]
    got = _run(lib, values=vals)
    assert got == {k: 0 for k in KINDS}
