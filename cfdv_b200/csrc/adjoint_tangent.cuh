// Directional derivative of the element residual r_e = rhs_e - R_e dU_e (the JVP), one lane per
// Gauss point (the kernel is in adjoint.cu; tests run the same code on the CPU with one fiber
// per lane).
//
// A warp takes EPW = 32 / Q elements (4 hex8, 8 quad4); lane = j * Q + q is Gauss point q of its
// element j, and also the element's node q.  With dU held fixed the residual of a pass is
//   r(N r) = sum_q [ sum_i omega dPhi_N,i Z_i(r) - omega Phi_N u0(r) - omega Psi_N qS(r) ],
//   Z_i = dt Fbar_i + dt (s1 a_i + s3 b_i) u0 + dt s3 sum_j c_ij u1_j - dt^2/2 (a_i + b_i) y,
//   y = divF + sum_j (s2 a_j + s4 b_j) u1_j,   qS = dt sum_i (s1 a_i + s3 b_i) uS   (2D domain)
// with u0, u1, uS the interpolated dU, its gradient and the sum of the gradient's components; on
// a face omega dPhi_N,i is -Phi_N en_i and the last two terms are absent (the regrouping of
// FDVGalerkin.h:405-451, 536-641, 643-756 in adjoint.cuh).  Every lane evaluates Z_i of its point
// in dual numbers along the tangent, once for the element's Ke rows, and the element's lanes
// exchange the derivatives through shared memory: lane N sums the rows of node N.
//
// Before, a thread evaluated the whole element functional for one row, so every Gauss point was
// evaluated Ke times: 14.1 ms for 24,576 hex8 elements.
#pragma once
#include "adjoint.cuh"

namespace cfdv {

template <int NDIM>
struct WarpJvp {
  using T = FormTraits<NDIM>;
  static constexpr int Q = T::Q, QF = T::QF, NNOD = T::NNOD, NBN = T::NBN, NEQ = T::NEQ, KE = T::KE,
                       NFACE = T::NFACE;
  static constexpr int EPW = 32 / Q;
  static_assert(Q == NNOD, "lane q owns Gauss point q and node q");
};

// what a lane hands to the node sums: omega dPhi_N,i (a face: -Phi_N en_i at the face's nodes),
// d Z_i(r), and in 2D omega Psi_N and qS with their derivatives; an odd number of doubles
template <int NDIM>
struct WarpJvpPoint {
  double wd[FormTraits<NDIM>::NNOD][NDIM];
  double dZ[NDIM][NDIM + 2];
  double psi[NDIM == 2 ? 4 : 1][2], qs[NDIM == 2 ? 4 : 1][2];
  double pad[NDIM == 2 ? 1 : 2];
};
static_assert((sizeof(WarpJvpPoint<2>) / 8) % 2 == 1 && (sizeof(WarpJvpPoint<3>) / 8) % 2 == 1, "bank spread");

template <int NDIM>
struct WarpJvpElem {
  using T = FormTraits<NDIM>;
  NodePrimT<Dual> nd[T::NNOD];
  double du[T::KE];
  Dual Mn[T::NNOD], Ren[T::NNOD], s[4];
};

template <int NDIM>
struct WarpJvpShared {
  WarpJvpElem<NDIM> el[WarpJvp<NDIM>::EPW];
  WarpJvpPoint<NDIM> pt[32];
};

// sum over r, c of one direction's 5 x 5 Jacobian block (row stride 5) times a vector
template <int NEQ, class V>
CFDV_HD CFDV_INLINE void jac_apply(const Dual* J, const Dual& f, const V* x, Dual* out) {
#pragma unroll
  for (int r = 0; r < NEQ; r++) {
    Dual t = 0.0;
#pragma unroll
    for (int c = 0; c < NEQ; c++) t += J[r * 5 + c] * x[c];
    out[r] += f * t;
  }
}

// y += s4 b_I u1_I (the a part is added for all directions at once, in jvp_point)
template <int NDIM, int I>
CFDV_HD CFDV_INLINE void jvp_beta(const GasT<Dual>& g, const GpStateT<Dual>& f, const Dual* s, const double (*u1)[5],
                                  Dual* y) {
  Dual J[25];
  jac_b_rows<NDIM>(g, f, I, J);
  jac_apply<NDIM + 2>(J, s[3], u1[I], y);
}

// Z_I but for the a part: dt Fbar_I + dt s3 (b_I u0 + sum_j c_Ij u1_j) - dt^2/2 b_I y
template <int NDIM, int I>
CFDV_HD CFDV_INLINE void jvp_z(const GasT<Dual>& g, const GpStateT<Dual>& f, const Dual& dt3, const Dual& mh2,
                               const double* u0, const double (*u1)[5], const Dual* y, Dual* Z) {
  constexpr int NEQ = NDIM + 2;
  {
    Dual J[25];
    jac_b_rows<NDIM>(g, f, I, J);
    jac_apply<NEQ>(J, dt3, u0, Z);
    jac_apply<NEQ>(J, mh2, y, Z);
  }
  Dual C[75];
  jac_c_rows<NDIM>(g, f, I, C);
#pragma unroll
  for (int j = 0; j < NDIM; j++) jac_apply<NEQ>(C + 25 * j, dt3, u1[j], Z);
}

// One Gauss point of a pass over the nodes pn[0..NN): d Z_i(r) into P.dZ, and in the 2D domain
// (uS set) qS into P.qs
template <int NDIM>
CFDV_HD CFDV_INLINE void jvp_point(const GasT<Dual>& g, const GpStateT<Dual>& f, const NodePrimT<Dual>* nd,
                                   const int* pn, int NN, const double* Phi, const double (*dPhi)[3], const Dual& dt,
                                   const Dual& dtsq_2, const Dual* s, const double* u0, const double (*u1)[5],
                                   const double* uS, bool withF, WarpJvpPoint<NDIM>& P) {
  constexpr int NEQ = NDIM + 2;
  Dual Z[NDIM][5], y[5];
  const Dual dt1 = dt * s[0], dt3 = dt * s[2], mh2 = -dtsq_2;
  // fluxes of the pass nodes: Z_i = dt Fbar_i, y = divF
  for (int i = 0; i < NDIM; i++)
    for (int r = 0; r < NEQ; r++) Z[i][r] = 0.0;
  for (int r = 0; r < NEQ; r++) y[r] = 0.0;
  for (int b = 0; b < NN; b++) {
    const NodePrimT<Dual>& nb = nd[pn[b]];
#pragma unroll
    for (int i = 0; i < NDIM; i++)
#pragma unroll
      for (int r = 0; r < NEQ; r++) {
        const Dual fg = node_flux_entry<NDIM>(f, nb, g.creyn, withF, i, r);
        Z[i][r] += Phi[b] * fg;
        y[r] += dPhi[b][i] * fg;
      }
  }
#pragma unroll
  for (int i = 0; i < NDIM; i++)
#pragma unroll
    for (int r = 0; r < NEQ; r++) Z[i][r] = dt * Z[i][r];
  // y += sum_j (s2 a_j + s4 b_j) u1_j
  Dual J[NDIM * 25];
  jac_a<NDIM>(g, f, J);
#pragma unroll
  for (int j = 0; j < NDIM; j++) jac_apply<NEQ>(J + 25 * j, s[1], u1[j], y);
  jvp_beta<NDIM, 0>(g, f, s, u1, y);
  jvp_beta<NDIM, 1>(g, f, s, u1, y);
  if constexpr (NDIM == 3) jvp_beta<NDIM, 2>(g, f, s, u1, y);
  // the a part of Z_i
#pragma unroll
  for (int i = 0; i < NDIM; i++) {
    jac_apply<NEQ>(J + 25 * i, dt1, u0, Z[i]);
    jac_apply<NEQ>(J + 25 * i, mh2, y, Z[i]);
  }
  if constexpr (NDIM == 2) {
    if (uS) {
      Dual qs[5];
      for (int r = 0; r < NEQ; r++) qs[r] = 0.0;
      for (int i = 0; i < NDIM; i++) {
        jac_apply<NEQ>(J + 25 * i, dt1, uS, qs);
        Dual B[25];
        jac_b_rows<NDIM>(g, f, i, B);
        jac_apply<NEQ>(B, dt3, uS, qs);
      }
      for (int r = 0; r < NEQ; r++) {
        P.qs[r][0] = qs[r].v;
        P.qs[r][1] = qs[r].d;
      }
    }
  }
  jvp_z<NDIM, 0>(g, f, dt3, mh2, u0, u1, y, Z[0]);
  jvp_z<NDIM, 1>(g, f, dt3, mh2, u0, u1, y, Z[1]);
  if constexpr (NDIM == 3) jvp_z<NDIM, 2>(g, f, dt3, mh2, u0, u1, y, Z[2]);
#pragma unroll
  for (int i = 0; i < NDIM; i++)
#pragma unroll
    for (int r = 0; r < NEQ; r++) P.dZ[i][r] = Z[i][r].d;
}

// The elements e0 .. e0 + EPW - 1 (those below n_elements): d r_e along (tU, t_dt, t_mach) into
// a.out; every lane of the warp calls it.  Lanes: sync(), any(p) as in adjoint_warp.cuh.
template <int NDIM, class Lanes>
CFDV_HD CFDV_INLINE void warp_jvp(const FunctionalArgs& a, WarpJvpShared<NDIM>& sh, int e0, int lane, Lanes& L) {
  using V = WarpJvp<NDIM>;
  constexpr int NNOD = V::NNOD, NEQ = V::NEQ, KE = V::KE, Q = V::Q, QF = V::QF, NBN = V::NBN;
  const int j = lane / Q, q = lane % Q, e = e0 + j;
  const bool valid = e < a.n_elements;
  WarpJvpElem<NDIM>& El = sh.el[j];
  WarpJvpPoint<NDIM>& P = sh.pt[lane];
  const GasT<Dual> g = dual_gas(a.gas, a.t_mach);
  const Dual dt(a.dt, a.t_dt), dtsq_2 = dt * dt / 2.0;
  const bool withF = (NDIM == 2) || a.physical_3d_flux;
  if (valid) {
    const int n = a.conn[(size_t)e * NNOD + q];
    Dual u[NEQ];
    for (int c = 0; c < NEQ; c++) u[c] = Dual(a.U[(size_t)n * NEQ + c], a.tU[(size_t)n * NEQ + c]);
    node_unpack<NDIM>(g, u, a.x + (size_t)n * NDIM, El.nd[q]);
    node_mach_re<NDIM>(g, El.nd[q], &El.Mn[q], &El.Ren[q]);
    for (int c = 0; c < NEQ; c++) El.du[q * NEQ + c] = a.dU[(size_t)n * NEQ + c];
  }
  L.sync();
  if (valid && q < 2) fdv_pair<NNOD>(q ? El.Ren : El.Mn, q, El.s);  // s1, s2 | s3, s4
  L.sync();
  const int hi = (valid && a.hnm_idx) ? a.hnm_idx[e] : -1;
  const double* Hn = (hi >= 0) ? a.hnm + (size_t)hi * NNOD * NNOD : nullptr;
  double row[NEQ];  // d r of node q
#pragma unroll
  for (int r = 0; r < NEQ; r++) row[r] = 0.0;
  // the passes: the domain (fc = -1), then each boundary face with 0 != bc < 100
  for (int fc = -1; fc < V::NFACE; fc++) {
    const bool face = fc >= 0;
    const int code = (face && valid) ? a.bc[(size_t)e * V::NFACE + fc] : 0;
    const bool pass = face ? (code != 0 && code < 100) : valid;
    if (face && !L.any(pass)) continue;
    if (pass && (!face || q < QF)) {
      double Phi[NNOD], dPhi[NNOD][3], en[3] = {0.0, 0.0, 0.0}, omega = 1.0;
      double jac[3][3];
      int pn[NNOD];
      const int NN = face ? NBN : NNOD;
      const NodePrimT<Dual>* all[NNOD];
      GpStateT<Dual> f;
      const double* x4[NNOD];
      for (int N = 0; N < NNOD; N++) x4[N] = El.nd[N].x;
      double z[3];
      if (!face) {
        double dPxi[NNOD][3], w = 1.0;
        for (int d = 0; d < NDIM; d++) {
          const int bit = (q >> (NDIM - 1 - d)) & 1;
          z[d] = a.gz[bit];
          w *= a.gw[bit];
        }
        shape_fn<NDIM>(z, Phi, dPxi);
        if (Hn) hnm_shape<NDIM>(Hn, Phi, dPxi);
        omega = w * phys_deriv<NDIM>(dPxi, El.nd, dPhi, jac);
        for (int N = 0; N < NNOD; N++) {
          pn[N] = N;
          all[N] = &El.nd[N];
        }
        gp_state_sums<NDIM, NNOD>(all, Phi, dPhi, f);
      } else {
        const double* xf[NBN];
        for (int i = 0; i < NBN; i++) {
          pn[i] = face_node(NDIM, fc, i);
          all[i] = &El.nd[pn[i]];
          xf[i] = x4[pn[i]];
        }
        double xl[4][3];
        if (NDIM == 3 && Hn) {  // adaptive element: face geometry from Hnm x
          const double* xe[8];
          for (int M = 0; M < 8; M++) xe[M] = x4[M % NNOD];
          hnm_face_nodes_3d(Hn, xe, fc, xl);
          for (int i = 0; i < NBN; i++) xf[i] = xl[i % 4];
        }
        face_point_geom<NDIM>(a.gz, a.gw, xf, q, Phi, dPhi, en);
        if constexpr (NDIM == 3)
          if (Hn) hnm_face_phi_3d(Hn, fc, Phi);
        gp_state_sums<NDIM, NBN>(all, Phi, dPhi, f);
      }
      f.mu = gas_mu(g, f.T);
      f.k = gas_k(g, f.mu);
      if (!face) {
        viscous_stress<NDIM>(f);
        if constexpr (NDIM == 2) {
          double pj[3][3];  // the upwind term's Jacobian: of the untransformed shape functions
          if (Hn) plain_jac_2d(z, x4, pj);
          Dual Psi[NNOD];
          psi_2d<Dual>(Hn ? pj : jac, x4, f, dPhi, Psi);
          for (int N = 0; N < NNOD; N++) {
            P.psi[N][0] = omega * Psi[N].v;
            P.psi[N][1] = omega * Psi[N].d;
          }
        }
      } else {
        for (int i = 0; i < NDIM; i++)
          for (int k = 0; k < NDIM; k++) f.tau[i][k] = 0.0;
        if constexpr (NDIM == 2)
          edit_face_state_2d(code, f, El.nd[face_node(NDIM, fc, 0)].x, El.nd[face_node(NDIM, fc, 1)].x, en);
        else
          edit_face_state_3d(code, f, en, a.gas.adiabatic);
      }
      double u0[5], u1[3][5], uS[5];
      for (int r = 0; r < NEQ; r++) {
        double b0 = 0.0, bs = 0.0, b1[3] = {0.0, 0.0, 0.0};
        for (int m = 0; m < NN; m++) {
          const double dv = El.du[pn[m] * NEQ + r];
          double sd = 0.0;
          b0 += Phi[m] * dv;
#pragma unroll
          for (int i = 0; i < NDIM; i++) {
            sd += dPhi[m][i];
            b1[i] += dPhi[m][i] * dv;
          }
          bs += sd * dv;
        }
        u0[r] = b0;
        uS[r] = bs;
        for (int i = 0; i < NDIM; i++) u1[i][r] = b1[i];
      }
      for (int N = 0; N < NNOD; N++)
        for (int i = 0; i < NDIM; i++) P.wd[N][i] = face ? 0.0 : omega * dPhi[N][i];
      if (face)
        for (int m = 0; m < NBN; m++)
          for (int i = 0; i < NDIM; i++) P.wd[pn[m]][i] = -(Phi[m] * en[i]);
      jvp_point<NDIM>(g, f, El.nd, pn, NN, Phi, dPhi, dt, dtsq_2, El.s, u0, u1, face ? nullptr : uS, withF, P);
    }
    L.sync();
    if (pass) {  // node q's rows: its sums over the element's points
      for (int p = 0; p < (face ? QF : Q); p++) {
        const WarpJvpPoint<NDIM>& O = sh.pt[j * Q + p];
#pragma unroll
        for (int r = 0; r < NEQ; r++) {
          double t = row[r];
#pragma unroll
          for (int i = 0; i < NDIM; i++) t += O.wd[q][i] * O.dZ[i][r];
          if constexpr (NDIM == 2)
            if (!face) t -= O.psi[q][1] * O.qs[r][0] + O.psi[q][0] * O.qs[r][1];
          row[r] = t;
        }
      }
    }
    L.sync();  // the points' slots are rewritten by the next pass
  }
  if (valid) {
    const uint64_t mask = a.rowmask ? a.rowmask[e] : 0ull;
#pragma unroll
    for (int r = 0; r < NEQ; r++)
      a.out[(size_t)e * KE + q * NEQ + r] = ((mask >> (q * NEQ + r)) & 1ull) ? 0.0 : row[r];
  }
  L.sync();  // the next elements may overwrite the shared state
}

}  // namespace cfdv
