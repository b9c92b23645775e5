"""Formation with node records (more than 4096 elements) and without, on both sides of the line:
sampled elements' matrices, rhs and FDV parameters against the oracle, 2D and 3D.  Bars as in the
other formation tests: 1e-12 of an element's largest entry, the parameters exact up to CUDA's pow
(2 ulp)."""
import numpy as np
import pytest

from conftest import elem_rel_err, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 64, 64, 0), (2, 66, 63, 0), (3, 16, 16, 16), (3, 17, 16, 16)])
def test_formation_on_both_sides_of_the_record_line(oracle_lib, shape):
    from cfdv_b200 import gpu as G, meshgen as mg
    nd, nx, ny, nz = shape
    case = mg.plate(nx, ny) if nd == 2 else mg.duct(nx, ny, nz)
    rng = np.random.default_rng(3)
    case.nodes[:, nd] *= 1.0 + 1e-2 * rng.standard_normal(case.n_nodes)
    o = oracle_lib.Oracle(case)
    U = o.init_U()
    with G.FDVSolver(case) as s:
        s.load_node_records()
        dt = s.cfl(0.5)
        s.form(dt, G.PREC_MIXED)
        R, rhs = s.element_matrices()
        par = s.fdv_params()
    Ro, ro = o.form(U, dt)
    assert elem_rel_err(R, Ro) <= 1e-12
    assert rel_err(rhs, ro) <= 1e-12
    assert np.abs(par - o.fdvparam(U)).max() <= 4.5e-16
