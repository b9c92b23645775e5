"""Hex8 formation on every boundary code: elements with none to three boundary faces, a random
state (all flux Jacobian rows, stress entries and c values non-zero), plain and hanging-node
elements, with and without the optional convective rhs flux; against the oracle, on the CPU (the
kernel's steps run thread by thread) and on the GPU.

Tolerance: an entry is a sum of 8 Gauss points x 4 coefficients of products with a handful of
roundings each, of terms up to about 10 times the element's largest entry here: 32 x ~10 x 1.1e-16
x 10 = 4e-13, held at 1e-12 as for the other formation tests."""
import numpy as np
import pytest

from conftest import elem_rel_err, rel_err
from test_form_emulated import emu, run_emu, _p  # noqa: F401  (fixture)

# 7 is left out: the oracle recomputes its stress once more than the kernel's edit does
CODES = [0, -12, -1, 1, 2, 4, 6, 8, 11, 12, 21, 22, 31, 32, 51, 77]


def case_for(code, adaptive, adiabatic):
    from cfdv_b200 import meshgen as mg
    c = mg.duct(3, 2, 2)
    rng = np.random.default_rng(100 + code)
    el = c.elements.copy()
    el[:, 8:][el[:, 8:] != 0] = code
    c.elements = el
    c.nodes[:, :3] += 0.02 * rng.standard_normal((c.n_nodes, 3))
    c.nodes[:, 3] = 1.0 + 0.2 * rng.random(c.n_nodes)
    c.nodes[:, 4:7] = rng.standard_normal((c.n_nodes, 3))
    c.nodes[:, 7] = 1.0 + 0.3 * rng.random(c.n_nodes)
    c.aero["Adiabatic"] = int(adiabatic)
    return mg.adaptive_demo(c) if adaptive else c


def expected(oracle_lib, c, phys):
    o = oracle_lib.Oracle(c)
    U = o.init_U()
    dt = o.cfl(U, 0.5)
    return o, U, dt, o.form(U, dt, apply_bc=True, physical_3d_flux=phys)


@pytest.mark.parametrize("adaptive,phys", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("code", CODES)
def test_boundary_codes_emulated(emu, oracle_lib, code, adaptive, phys):  # noqa: F811
    c = case_for(code, adaptive, adiabatic=code % 2)
    o, U, dt, (Ro, ro) = expected(oracle_lib, c, phys)
    if adaptive:
        idx = np.ascontiguousarray(c.hnm_index(), np.int32)
        hnm = np.ascontiguousarray(np.transpose(c.adap_hnm, (0, 2, 1)), np.float64)
        emu.emu_set_adaptive(_p(idx), _p(hnm))
    try:
        bad, R, R32, rhs, _ = run_emu(emu, c, U, dt, o.rowmask(), int(phys))
    finally:
        emu.emu_set_adaptive(None, None)
    assert bad == 0
    assert elem_rel_err(R, Ro) <= 1e-12
    assert rel_err(rhs, ro) <= 1e-12
    np.testing.assert_array_equal(R32, R.astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("adaptive,phys", [(False, False), (False, True), (True, False)])
@pytest.mark.parametrize("code", CODES)
def test_boundary_codes_gpu(oracle_lib, code, adaptive, phys):
    from cfdv_b200 import gpu as G
    c = case_for(code, adaptive, adiabatic=code % 2)
    _, _, dt, (Ro, ro) = expected(oracle_lib, c, phys)
    with G.FDVSolver(c, physical_3d_flux=phys) as s:
        s.load_node_records()
        s.form(dt)
        R, rhs = s.element_matrices()
    assert elem_rel_err(R, Ro) <= 1e-12
    assert rel_err(rhs, ro) <= 1e-12
