"""Solves whose Krylov basis is streamed through the shared-memory ring, on meshes whose blocks own
one, two and three chunks of unknowns, both precisions, with and without the preconditioner: the
same matrices give the same bits every time (a slot handed back before its values were read showed
as last-bit differences between repeats from three chunks on), and the solution has the residual
that the solve reports."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,precond", [((34, 30, 18), True), ((44, 40, 24), False), ((60, 55, 35), True),
                                            ((97, 53, 29), True)])
def test_streamed_solve_repeats_bit_for_bit(shape, precond, precision):
    from cfdv_b200 import gpu as G, meshgen as mg
    case = mg.duct(*shape)
    rng = np.random.default_rng(1)
    case.nodes[:, 3] *= 1.0 + 1e-3 * rng.standard_normal(case.n_nodes)
    prec = G.PREC_MIXED if precision == "mixed" else G.PREC_FP64
    with G.FDVSolver(case) as s:
        s.load_node_records()
        s.form(s.cfl(0.5), prec)
        b = s.rhs_vector()
        first = None
        for _ in range(6):
            rep = s.gmres(mode=G.GMRES_CORRECT, m=40, restarts=30, rtol=1e-8, precision=prec, precond=precond)
            du = s.du()
            if first is None:
                first = du
                res = np.linalg.norm(b - s.matvec(du)) / np.linalg.norm(b)
                # the two residuals sum the same terms in other orders: below 1e-12 of ||b|| apart
                assert abs(res - rep["true_rel_res"]) <= 1e-12
            np.testing.assert_array_equal(du, first)
