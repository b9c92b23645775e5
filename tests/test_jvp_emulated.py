"""The JVP with one lane per Gauss point (cfdv_b200/csrc/adjoint_tangent.cuh) against the
forward-mode functional evaluated row by row, on every element of the small cases, hanging-node
ones and the optional 3D convective flux included: on the CPU (lanes as fibers) and on the GPU.

Tolerance: both evaluate the same dual-number physics and differ in the order of sums of about
100 terms, bounded by 100 x 1.1e-16 of the largest term: 1e-13 of the largest entry on the CPU
(a state's terms exceed the result by less than 10), 1e-10 on the GPU, whose libm differs, as for
the other adjoint kernels (the lid's test function cancels to a few digits there: 1e-3)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ADAPTIVE_CASES, ROOT, SMALL_CASES
from test_adjoint_emulated import Setup, _p, emu  # noqa: F401  (fixture)

EMU = os.path.join(ROOT, "tests", "emu", "libjvp_emu.so")
CSRC = os.path.join(ROOT, "cfdv_b200", "csrc")


@pytest.fixture(scope="module")
def jvp_emu():
    src = os.path.join(ROOT, "tests", "emu", "jvp_emu.cpp")
    deps = [src] + [os.path.join(CSRC, f) for f in ("adjoint.cuh", "adjoint_tangent.cuh", "dual.cuh", "formation.cuh",
                                                     "fdv_physics.cuh", "cfdv_types.h")]
    if not os.path.exists(EMU) or os.path.getmtime(EMU) < max(os.path.getmtime(f) for f in deps):
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread", "-Wno-unknown-pragmas", src, "-o",
                        EMU], check=True)
    L = C.CDLL(EMU)
    P, D, I = C.c_void_p, C.c_double, C.c_int
    L.emu_functional.argtypes = [I, I, P, P, P, P, P, D, D, D, D, D, D, I, D, I, I, P, P, P, D, D, P, P]
    L.emu_jvp_warp.argtypes = [I, I, P, P, P, P, P, D, D, D, D, D, D, I, D, I, P, P, D, D, P]
    L.emu_set_adaptive.argtypes = [P, P]
    return L


def tangent(s):
    rng = np.random.default_rng(5)
    return rng.standard_normal(s.o.n_dof) * 1e-3, 0.3 * s.dt, 0.02


@pytest.mark.parametrize("phys", [0, 1])
@pytest.mark.parametrize("name", SMALL_CASES + ADAPTIVE_CASES)
def test_warp_jvp_matches_row_by_row(jvp_emu, oracle_lib, name, phys):
    s = Setup(oracle_lib, name)
    if phys and s.case.ndim == 2:
        pytest.skip("the 3D flux switch has no effect in 2D")
    tU, tdt, tM = tangent(s)
    s.arm(jvp_emu)
    args = (s.case.ndim, s.E, _p(s.U), _p(s.x), _p(s.conn), _p(s.bc), _p(s.mask), *s.gas, s.dt, phys)
    ref, val, out = np.zeros(s.E * s.Ke), np.zeros(s.E), np.zeros(s.E * s.Ke)
    jvp_emu.emu_functional(*args, 1, _p(s.du), _p(s.w), _p(tU), tdt, tM, _p(ref), _p(val))
    jvp_emu.emu_jvp_warp(*args, _p(s.du), _p(tU), tdt, tM, _p(out))
    assert np.abs(ref).max() > 0
    assert np.abs(out - ref).max() <= 1e-13 * np.abs(ref).max()


@pytest.mark.gpu
@pytest.mark.parametrize("name", SMALL_CASES + ADAPTIVE_CASES)
def test_gpu_jvp_matches_row_by_row(emu, oracle_lib, name):  # noqa: F811
    from cfdv_b200 import gpu as G
    s = Setup(oracle_lib, name)
    tU, tdt, tM = tangent(s)
    ref, _ = s.emu(emu, mode=1, tU=tU, tdt=tdt, tM=tM)
    want = s.o.compose_rhs(ref)
    with G.FDVSolver(s.case) as g:
        g.load_node_records()
        g.set_state(s.U)
        g.form(s.dt)
        got = g.jvp(s.du, tU, t_dt=tdt, t_mach=tM)
    assert np.abs(got - want).max() <= (1e-3 if name.startswith("lid") else 1e-10) * np.abs(want).max()
