"""The VJP and JVP kernels take more dynamic shared memory than a launch may have by default.  The
limit that allows it belongs to a device's context, so it has to be raised there and not once per
process: a second device, or the same device after cudaDeviceReset, starts with the default again.
One device shows it with a reset; a second one is tried as well where the machine has one."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

_CHILD = r"""
import ctypes as C, sys
import numpy as np
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from conftest import get_case
from cfdv_b200 import gpu as G
G.lib()  # loads the CUDA runtime that the library is linked with
rt = C.CDLL("libcudart.so.12")

def products(name):
    case = get_case(name)
    rng = np.random.default_rng(4)
    with G.FDVSolver(case) as s:
        s.load_node_records()
        s.form(s.cfl(float(case.control["cfl"])))
        du, t, w = (rng.standard_normal(s.n_dof) for _ in range(3))
        return s.jvp(1e-3 * du, 1e-3 * t, t_dt=1e-4, t_mach=1e-3), s.vjp(w, 1e-3 * du)[0]

def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))

first = {n: products(n) for n in ("plate20", "duct4")}
count = C.c_int()
assert rt.cudaGetDeviceCount(C.byref(count)) == 0
if count.value > 1:
    assert rt.cudaSetDevice(1) == 0
    assert all(same(products(n), first[n]) for n in first), "second device"
    assert rt.cudaSetDevice(0) == 0
assert rt.cudaDeviceReset() == 0
assert all(same(products(n), first[n]) for n in first), "after a reset"
print("equal")
"""


def test_products_run_in_every_context_of_a_process():
    r = subprocess.run([sys.executable, "-c", _CHILD, ROOT], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and r.stdout.strip() == "equal", r.stderr[-2000:]
