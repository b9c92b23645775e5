"""Boundary code 7 on hex8 faces.  The reference's case has no break: it runs on into the body of codes
77 and 32 (eval2dboundary.h:113-145), which forms the stress once more, so of the two stress columns
that were set to zero the first one comes back.  The formation, the VJP and the JVP share the edit.

Element matrices against the oracle: the tolerance of the other boundary codes (test_form_hex.py).
Derivatives along a direction of the state's own size: a central difference with step h = 1e-5 carries
about 1e2 x 1e-16 / h = 1e-9 of rounding and a few h^2 of truncation, held at 1e-6.  VJP and JVP are
transposes of each other to rounding, 1e-10 as for the other adjoint kernels."""
import numpy as np
import pytest

from conftest import elem_rel_err, rel_err
from test_adjoint_emulated import Setup, emu as adj_emu  # noqa: F401  (fixture)
from test_form_emulated import _p, emu, run_emu  # noqa: F401  (fixture)
from test_form_hex import case_for, expected

VARIANTS = [(False, False), (False, True), (True, False)]


@pytest.mark.parametrize("adaptive,phys", VARIANTS)
def test_formation_emulated(emu, oracle_lib, adaptive, phys):  # noqa: F811
    c = case_for(7, adaptive, adiabatic=True)
    o, U, dt, (Ro, ro) = expected(oracle_lib, c, phys)
    if adaptive:
        idx = np.ascontiguousarray(c.hnm_index(), np.int32)
        hnm = np.ascontiguousarray(np.transpose(c.adap_hnm, (0, 2, 1)), np.float64)
        emu.emu_set_adaptive(_p(idx), _p(hnm))
    try:
        bad, R, _, rhs, _ = run_emu(emu, c, U, dt, o.rowmask(), int(phys))
    finally:
        emu.emu_set_adaptive(None, None)
    assert bad == 0
    assert elem_rel_err(R, Ro) <= 1e-12
    assert rel_err(rhs, ro) <= 1e-12


class Code7(Setup):
    """The random state of case_for(7) in the form that the adjoint's emulation takes."""

    def __init__(self, O):
        self.case = c = case_for(7, False, adiabatic=True)
        self.o = o = O.Oracle(c)
        self.U = o.init_U()
        self.dt = o.cfl(self.U, 0.5)
        rng = np.random.default_rng(3)
        self.du = 1e-3 * rng.standard_normal(o.n_dof)
        self.w = rng.standard_normal(o.n_dof)
        self.tU = rng.standard_normal(o.n_dof)
        self.mask = o.rowmask()
        self.x = np.ascontiguousarray(c.nodes[:, :3])
        self.conn = np.ascontiguousarray(c.conn, np.int32)
        self.bc = np.ascontiguousarray(c.bc, np.int32)
        a = c.aero
        self.gas = (float(a["gamma"]), float(a["M"]), float(a["Re"]), float(a["Pr"]), float(a["Tinf"]),
                    float(a["Twall"]), int(a["Adiabatic"]))
        self.E, self.Ke = c.n_elements, o.Ke
        self.hidx = self.hnm = None


def test_derivatives_emulated(adj_emu, oracle_lib):  # noqa: F811
    """sum_e dL_e/dU . t of the reverse sweep's seeds against differences of the oracle's residual."""
    s = Code7(oracle_lib)
    assert (s.bc == 7).any()
    g, val = s.emu(adj_emu)
    ref = s.oracle_L()
    assert np.abs(val - ref).max() <= 1e-12 * np.abs(ref).max()
    t = s.tU * np.abs(s.U)
    h = 1e-5
    fd = (s.oracle_L(U=s.U + h * t) - s.oracle_L(U=s.U - h * t)) / (2 * h)
    got = np.array([g[e, : s.Ke] @ t[s.idx(e)] for e in range(s.E)])
    assert np.abs(got - fd).max() <= 1e-6 * np.abs(fd).max()


@pytest.mark.gpu
@pytest.mark.parametrize("adaptive,phys", VARIANTS)
def test_formation_gpu(oracle_lib, adaptive, phys):
    from cfdv_b200 import gpu as G
    c = case_for(7, adaptive, adiabatic=True)
    _, _, dt, (Ro, ro) = expected(oracle_lib, c, phys)
    with G.FDVSolver(c, physical_3d_flux=phys) as s:
        s.load_node_records()
        s.form(dt)
        R, rhs = s.element_matrices()
    assert elem_rel_err(R, Ro) <= 1e-12
    assert rel_err(rhs, ro) <= 1e-12


@pytest.mark.gpu
def test_products_gpu(oracle_lib):
    from cfdv_b200 import gpu as G
    s = Code7(oracle_lib)
    with G.FDVSolver(s.case) as g:
        g.load_node_records()
        g.form(s.dt)
        jt = g.jvp(s.du, s.tU)
        gU, _, _ = g.vjp(s.w, s.du)
    lhs, rhs = float(s.w @ jt), float(gU @ s.tU)
    terms = float(np.abs(s.w) @ np.abs(jt)) + float(np.abs(gU) @ np.abs(s.tU))
    assert abs(lhs - rhs) <= 1e-10 * terms
