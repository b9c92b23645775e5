"""Contexts of different meshes in several host threads at once: a context belongs to one thread, so each
thread has its own, and every solve must give what it gives alone.  The meshes need different amounts of
shared memory for the same solve kernel, whose limit is a property of the kernel and not of a launch."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solves(case, mode, count):
    from cfdv_b200 import gpu as G
    opts = dict(mode=G.GMRES_REFERENCE, m=20, restarts=1) if mode == "reference" else dict(
        mode=G.GMRES_CORRECT, m=20, restarts=20, rtol=1e-8)
    with G.FDVSolver(case) as s:
        s.load_node_records()
        s.form(s.cfl(0.5))
        out = []
        for _ in range(count):
            s.gmres(**opts)
            out.append(s.du())
    return out


@pytest.mark.parametrize("mode", ["reference", "correct"])
def test_solves_in_threads_match_solves_alone(mode):
    from cfdv_b200 import meshgen as mg
    cases = [mg.lid(8), mg.lid(48), mg.lid(24)]
    want = [solves(c, mode, 1)[0] for c in cases]
    got, errors = [None] * len(cases), []

    def work(k):
        try:
            got[k] = solves(cases[k], mode, 300)
        except Exception as e:  # a refused launch
            errors.append(f"{k}: {e}")

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, g in zip(want, got):
        for du in g:
            np.testing.assert_array_equal(du, w)
