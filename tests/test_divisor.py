"""The division by a shared value (cfdv_b200/csrc/divisor.h) against IEEE division, on the CPU: the last
bit may differ for ordinary numbers, nothing else does.  With q = x RN(1/d) off by at most 1.5 ulp, the
residual x - q d is exact in one fused operation and its correction leaves less than one ulp, so the
result is the rounded quotient or its neighbour.  Where a product would overflow, lose bits to subnormal
numbers or meet an infinity, and for zeros, the quotient is the division's."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

EMU = os.path.join(ROOT, "tests", "emu", "libdiv_emu.so")


@pytest.fixture(scope="module")
def divide():
    src = os.path.join(ROOT, "tests", "emu", "div_emu.cpp")
    hdr = os.path.join(ROOT, "cfdv_b200", "csrc", "divisor.h")
    if not os.path.exists(EMU) or os.path.getmtime(EMU) < max(os.path.getmtime(src), os.path.getmtime(hdr)):
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", src, "-o", EMU], check=True)
    L = C.CDLL(EMU)
    L.emu_divide.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_long]

    def f(x, d):
        x, d = (np.ascontiguousarray(v, np.float64) for v in np.broadcast_arrays(x, d))
        q = np.empty_like(x)
        L.emu_divide(x.ctypes.data, d.ctypes.data, q.ctypes.data, q.size)
        with np.errstate(all="ignore"):
            return q, x / d
    return f


SPECIAL = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 3e-310, 2.3e-308, 1e-300, 1e-290, 1e-200, 1e-139, 1.0,
           -3.0, 1e139, 1e200, 1e290, 1e300, 1.7976931348623157e308]


def test_ordinary_numbers_to_the_last_bit(divide):
    rng = np.random.default_rng(11)
    x = rng.standard_normal(400_000) * 10.0 ** rng.uniform(-30, 30, 400_000)
    d = rng.standard_normal(400_000) * 10.0 ** rng.uniform(-30, 30, 400_000)
    q, want = divide(x, d)
    assert (np.abs(q - want) <= np.spacing(np.abs(want))).all()


@pytest.mark.parametrize("d", [v for v in SPECIAL if v != 0.0] + [0.0, 7.0, 1.0 / 3.0, 7e-13])
def test_special_numerators(divide, d):
    q, want = divide(np.array(SPECIAL), d)
    np.testing.assert_array_equal(np.isnan(q), np.isnan(want))
    ok = ~np.isnan(want)
    np.testing.assert_array_equal(np.signbit(q[ok]), np.signbit(want[ok]))
    np.testing.assert_array_equal(np.isinf(q[ok]), np.isinf(want[ok]))
    fin = ok & np.isfinite(want)
    normal = fin & (np.abs(want) >= 2.3e-308)
    assert (np.abs(q[normal] - want[normal]) <= np.spacing(np.abs(want[normal]))).all()
    np.testing.assert_array_equal(q[fin & ~normal], want[fin & ~normal])


def test_subnormal_quotients(divide):
    rng = np.random.default_rng(12)
    x = rng.uniform(1, 2, 20_000) * 10.0 ** rng.uniform(-308, -200, 20_000)
    d = rng.uniform(1, 2, 20_000) * 10.0 ** rng.uniform(0, 110, 20_000)
    q, want = divide(x, d)
    low = np.abs(want) < 2.3e-308
    assert low.any()
    np.testing.assert_array_equal(q[low], want[low])
