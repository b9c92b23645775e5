"""The reference-mode solve as one persistent launch per restart cycle (m + 2 <= 64) and as one
launch per Gram-Schmidt pass (larger m), against the oracle's restatement of MPI_GMRES::iterate:
restart lengths at the ends of both ranges, cycles that run to m and cycles that the estimate ends,
one and three restarts, 2D and 3D.

Bars: the estimates to 1e-10 of the first one, as for the golden histories; dU to 1e-7 of its
largest entry, because the reference's near-diagonal back substitution multiplies the rounding of
the Hessenberg entries (about 1e-14) by quotients of them, up to 1e6 here."""
import numpy as np
import pytest

from conftest import get_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["lid8", "plate20", "ramp4", "duct4"])
@pytest.mark.parametrize("m,restarts", [(1, 1), (2, 3), (20, 1), (20, 3), (62, 1), (63, 1), (70, 2)])
def test_reference_cycle_matches_oracle(oracle_lib, name, m, restarts):
    from cfdv_b200 import gpu as G
    case = get_case(name)
    o = oracle_lib.Oracle(case)
    U = o.init_U()
    with G.FDVSolver(case) as s:
        s.load_node_records()
        dt = s.cfl(float(case.control["cfl"]))
        s.form(dt)
        R, rhs = s.element_matrices()
        rep = s.gmres(mode=G.GMRES_REFERENCE, m=m, restarts=restarts)
        du = s.du()
        s.update()
        assert rel_err(s.get_state(), U + du) == 0.0
    du_o, rep_o = o.gmres_ref(R, rhs, m, restarts)
    assert rep["restarts"] == restarts
    assert rep["est"].shape == rep_o["est"].shape
    assert np.abs(rep["est"] - rep_o["est"]).max() <= 1e-10 * np.abs(rep_o["est"]).max()
    assert rep["matvecs"] == restarts + len(rep["est"])
    assert rel_err(du, du_o) <= 1e-7
