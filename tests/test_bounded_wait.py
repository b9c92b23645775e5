"""The waits of the persistent solve's shared-memory rings (cfdv_b200/csrc/bounded_wait.h) on the
CPU, the lanes of a warp as threads.  In a failing launch the lanes see the failure mark, the clock
and the end of the phase at different polls; they must leave with one answer, because the code behind
the wait is warp-wide, and a copy in flight must still be waited for."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

EMU = os.path.join(ROOT, "tests", "emu", "libwait_emu.so")
THREAD, WARP, LANDED = 0, 1, 2
NEVER = -1


@pytest.fixture(scope="module")
def emu():
    src = os.path.join(ROOT, "tests", "emu", "wait_emu.cpp")
    hdr = os.path.join(ROOT, "cfdv_b200", "csrc", "bounded_wait.h")
    if not os.path.exists(EMU) or os.path.getmtime(EMU) < max(os.path.getmtime(src), os.path.getmtime(hdr)):
        subprocess.run(["g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-pthread", src, "-o", EMU], check=True)
    L = C.CDLL(EMU)
    L.emu_wait.argtypes = [C.c_int, C.c_void_p, C.c_void_p, C.c_ulonglong, C.c_void_p, C.c_void_p]
    return L


def wait(emu, kind, done_at, failing_at, ns=1000):
    d = np.ascontiguousarray(np.broadcast_to(done_at, 32), np.int64)
    f = np.ascontiguousarray(np.broadcast_to(failing_at, 32), np.int64)
    ans, marked = np.zeros(32, np.int32), np.zeros(32, np.int32)
    emu.emu_wait(kind, d.ctypes.data, f.ctypes.data, ns, ans.ctypes.data, marked.ctypes.data)
    return ans, marked


@pytest.mark.parametrize("done_at", [0, 1, 100, 5000])
def test_a_finished_phase_is_seen(emu, done_at):
    for kind in (THREAD, WARP, LANDED):
        ans, marked = wait(emu, kind, done_at, NEVER)
        assert ans.all() and not marked.any()


@pytest.mark.parametrize("done_at", [100, 640, 5000])
@pytest.mark.parametrize("failing_at", [[64 * (k + 1) for k in range(32)], [64] + [NEVER] * 31, [NEVER] * 31 + [64]])
def test_lanes_leave_with_one_answer(emu, done_at, failing_at):
    """Some lanes see the mark before the phase ends and some the phase first."""
    alone, _ = wait(emu, THREAD, done_at, failing_at)
    together, _ = wait(emu, WARP, done_at, failing_at)
    assert (together == alone.min()).all()


def test_time_limit_marks_the_launch(emu):
    for kind in (THREAD, WARP, LANDED):
        ans, marked = wait(emu, kind, NEVER, NEVER, ns=1_000_000)  # 2 s pass after 2000 polls
        assert not ans.any() and marked.all()


@pytest.mark.parametrize("done_at", [65, 1000, 100_000])
def test_a_copy_in_flight_is_waited_for_in_a_failing_launch(emu, done_at):
    assert not wait(emu, THREAD, done_at, 0)[0].any()  # any other wait gives up
    ans, marked = wait(emu, LANDED, done_at, 0)
    assert ans.all() and not marked.any()


def test_the_kernel_waits_this_way():
    """Consumers wait as a warp, and the two drains of the producers for what has been issued."""
    with open(os.path.join(ROOT, "cfdv_b200", "csrc", "gmres_persistent.cu")) as f:
        src = f.read()
    body = src[src.index("elem_pass_ring("):src.index("// Element pass Y_e = R_e x_e")]
    waits = [ln.strip() for ln in body.splitlines() if "mbar_wait" in ln]
    assert len(waits) == 8
    for ln in waits:
        empty = ".empty" in ln  # the producer, one thread
        leaves = "return" in ln
        assert ("mbar_wait_thread(" in ln) == empty
        assert ("mbar_wait_warp(" in ln) == (not empty and leaves)
        assert ("mbar_wait_landed(" in ln) == (not empty and not leaves)
