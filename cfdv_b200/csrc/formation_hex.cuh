// FDV element formation of a hex8 element (3D) as the steps of one 128-thread block.
//
// The element matrix is a sum over Gauss points of a contraction
//   R(N r, M s) = sum_q sum_c G_c(N; r, s) B_c(M),   B = (Phi_M, dPhi_M,x, dPhi_M,y, dPhi_M,z),
//   G_c(N; r, s) = sum_k A_k(N) T_ck(r, s),          A = wJ (Phi_N, dPhi_N,x, dPhi_N,y, dPhi_N,z),
// with T_00 = delta_rs, T_0,1+i = -X_i, T_1+j,1+i = h_ij (FDVGalerkin.h:405-451; X_i =
// dt (s1 a_i + s3 b_i), h_ij = -dt s3 c_ij + dt^2/2 A_i D_j, A = a + b, D = s2 a + s4 b).
// A boundary face adds the same sum over its points with A = -Phi_N (0, en) (X_i enters with
// +en_i and m_ij = -h_ij, FDVGalerkin.h:455-533, 643-756).
//
// Both sums and the products A_i D_j are small dense products, so they run on the FP64 matrix instruction (mma m8n8k4).  On the B200 it has the rate of the
// FP64 FMA pipe (37 TFLOP/s measured for both) but takes 1 issue slot and 1 + 1 operand loads
// for 256 multiply-adds, where the scalar form took 8 and one shared-memory load per 1.5 of
// them; the earlier scalar kernel was bound by issue and shared-memory loads (46% of the issue
// slots, 20% of the FP64 pipe).  Formation of the 128x64x32 ramp (262,144 elements, FP64 and FP32
// copies): 10.9 -> 4.7 ms; of 2,275 elements 171 -> 94 us.  By step, of 65,536 elements alone: up
// to the Jacobian rows 0.49 ms, h 0.14, the contraction 0.30 (its 312 products an element at the
// matrix rate: 0.29), the store 0.13, boundary faces 0.19.  The result of the G product is, lane by lane, the A operand
// of the second one: the G tile's columns are ordered (c, r s parity), so no lane moves data.
//
// The flux Jacobians are evaluated by row: one thread per (Gauss point, direction i, row r) has
// the row of a_i and b_i from direction-generic formulas (all threads of a warp run the same
// code) and stores X, A and D at once.  c_ij has 31 distinct non-zero values per Gauss point;
// they are tabulated and the h product starts from them.
//
// Every step is a function of (block state, thread), so tests run the same code thread by
// thread on the CPU; there the matrix products are scalar loops over the same operands.
#pragma once

namespace cfdv {

// ---- 8 x 8 x 4 FP64 product: lane holds c(N, n0), c(N, n0 + 1), N = lane / 4, n0 = 2 (lane % 4);
// A(row, k) and B(k, col) read the operands ------------------------------------------------
template <class FA, class FB>
CFDV_HD CFDV_INLINE void mma_f64(int lane, FA A, FB B, double& c0, double& c1) {
#ifdef __CUDA_ARCH__
  const double a = A(lane >> 2, lane & 3), b = B(lane & 3, lane >> 2);
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
#else
  for (int k = 0; k < 4; k++) {
    c0 += A(lane >> 2, k) * B(k, 2 * (lane & 3));
    c1 += A(lane >> 2, k) * B(k, 2 * (lane & 3) + 1);
  }
#endif
}

// the product alone: c = A B
template <class FA, class FB>
CFDV_HD CFDV_INLINE void mma_f64_fresh(int lane, FA A, FB B, double& c0, double& c1) {
#ifdef __CUDA_ARCH__
  const double a = A(lane >> 2, lane & 3), b = B(lane & 3, lane >> 2), z = 0.0;
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %4};"
      : "=d"(c0), "=d"(c1)
      : "d"(a), "d"(b), "d"(z));
#else
  c0 = c1 = 0.0;
  mma_f64(lane, A, B, c0, c1);
#endif
}

// ---- the distinct values of c_ij (1/Re folded in) -----------------------------------------
// With M = mu / (rho Re), L = -2/3 M, K = k / (Cv rho Re), w = momentum / rho, W2 = w.w (k, l < 3):
//   c_ij(1+k, 1+l) = -(M (d_ij d_kl + d_il d_jk) + L d_ik d_jl)
//   c_ij(1+k, 0)   =   M (d_ij w_k + d_jk w_i) + L d_ik w_j
//   c_ij(4, 1+l)   = -(M (d_ij w_l + d_il w_j) + L d_jl w_i) + d_ij K w_l
//   c_ij(4, 0)     =   M (d_ij W2 + w_i w_j) + L w_i w_j - d_ij K (W2 - E),   c_ij(4, 4) = -d_ij K
// (NavierStokes3D.h:347-477 written for a general direction).  Table slots of the values:
enum HexC : int {
  HC_NMR = 0,   // -(2M + L)
  HC_NM = 1,    // -M
  HC_NL = 2,    // -L
  HC_NK = 3,    // -K
  HC_MRW = 4,   // (2M + L) w_l
  HC_MW = 7,    // M w_l
  HC_LW = 10,   // L w_l
  HC_KMRW = 13, // (K - 2M - L) w_l
  HC_KMW = 16,  // (K - M) w_l
  HC_NMW = 19,  // -M w_l
  HC_NLW = 22,  // -L w_l
  HC_EE = 25,   // c_ii(4, 0)
  HC_WW = 28,   // (M + L) w_a w_b for the pairs (0,1), (0,2), (1,2)
  HC_ZERO = 31,
  HC_COUNT = 32
};
constexpr int hex_c_slot(int i, int r, int j, int s) {
  if (r == 0 || i > 2 || j > 2) return HC_ZERO;
  if (s == 4) return (r == 4 && i == j) ? HC_NK : HC_ZERO;
  const int k = r - 1, l = s - 1;
  if (r < 4 && s > 0) {
    if (i == j) return k != l ? HC_ZERO : (k == i ? HC_NMR : HC_NM);
    return (l == i && k == j) ? HC_NM : ((k == i && l == j) ? HC_NL : HC_ZERO);
  }
  if (r < 4) {  // s == 0
    if (i == j) return k == i ? HC_MRW + i : HC_MW + k;
    return k == j ? HC_MW + i : (k == i ? HC_LW + j : HC_ZERO);
  }
  if (s > 0) {  // r == 4
    if (i == j) return l == i ? HC_KMRW + i : HC_KMW + l;
    return l == i ? HC_NMW + j : (l == j ? HC_NLW + i : HC_ZERO);
  }
  return i == j ? HC_EE + i : HC_WW + (i + j - 1);
}
// per lane, the slots of its 8 entries of the h product, one byte each: entry (mt, nt, e) of
// byte 4 mt + 2 nt + e is row 8 mt + lane / 4 = 5 i + r, column 8 nt + 2 (lane % 4) + e = 5 j + s
struct HexCTable {
  unsigned long long v[32];
};
constexpr HexCTable make_hex_c_table() {
  HexCTable t{};
  for (int lane = 0; lane < 32; lane++) {
    unsigned long long w = 0;
    for (int b = 0; b < 8; b++) {
      const int row = 8 * (b >> 2) + lane / 4, col = 8 * ((b >> 1) & 1) + 2 * (lane % 4) + (b & 1);
      const int slot = (row < 15 && col < 15) ? hex_c_slot(row / 5, row % 5, col / 5, col % 5) : (int)HC_ZERO;
      w |= (unsigned long long)slot << (8 * b);
    }
    t.v[lane] = w;
  }
  return t;
}
#if defined(__CUDACC__)
__device__
#endif
static constexpr HexCTable kHexCTable = make_hex_c_table();

// ---- block state --------------------------------------------------------------------------
constexpr int kHexNodeLd = 12;  // node fields E, T, U[5], v[3], 1, p
constexpr int kHexTileLd = 42;  // column stride of the element-matrix tile (bank-conflict free)
constexpr int kHexTLd = 312;    // T of a Gauss point: (r s, c, i) at (5 r + s) * 12 + 3 c + i, and one entry of room

struct HexGp {  // one Gauss point; an odd number of doubles
  GpState st;           // flow state (edited on boundary faces)
  double S[4];          // sum_b Phi_b, sum_b dPhi_b,i
  double raw[4][3];     // sum_b Phi_b v_b, sum_b dPhi_b,i v_b (as interpolated)
  double irho, w[3], divm, vgr, q2;  // 1/rho, momentum/rho, div(momentum), v.grad(rho), v.v
  double ctab[HC_COUNT];             // -dt s3 c values
  double divF[5];
  double A[16][5];      // dt^2/2 A_i(r, .) in row 5 i + r
  double D[4][20];      // D_j(1+k, s) at [k][5 j + s]
  double pad;
};
static_assert(sizeof(GpState) == 48 * sizeof(double) && (sizeof(HexGp) / sizeof(double)) % 2 == 1, "HexGp layout");

template <>
struct FormShared<3> {
  double T[8][kHexTLd];          // of the domain points; a face uses points 0-3
  double F[8 * kHexNodeLd];      // node fields
  double x[8][3];
  double cM[8][33];              // coefficient rows (N, c) at 4 N + c of the points of a pass
  double wJ[8];
  double en[4][3];               // weighted normals of a face's points
  double P[8][16];               // dt Fbar(i, r) - dt^2/2 sum_s A_i(r, s) divF(s) at 5 i + r
  double rhs[40];
  double Mn[8], Ren[8];
  double s[4], dt, dtsq_2, reinv, rCv;  // reinv = 1 / Re, rCv = 1 / Cv
  double delta[26 * 4];          // T_c0 of the entries: delta_rs at c = 0
  uint64_t mask;
  int faces[6], codes[6], nfaces, hnm;
  union {
    HexGp gp[8];
    double jac[8][9];
    double Rt[40 * kHexTileLd];  // element matrix, column-major; from the domain contraction on
  };
};
static_assert(4 * sizeof(HexGp) <= 4 * kHexTLd * sizeof(double), "a face's points fit in T's second half");

// A face's points are evaluated while the tile is live: they borrow T of points 4-7
template <bool FACE>
CFDV_HD CFDV_INLINE HexGp& hex_gp(FormShared<3>& sh, int q) {
  return FACE ? reinterpret_cast<HexGp*>(&sh.T[4][0])[q] : sh.gp[q];
}

// ---- steps ---------------------------------------------------------------------------------
// load: node records, boundary faces, FDV parameters, shape functions and natural derivatives (q, N)
CFDV_HD CFDV_INLINE void hex_load(const FormArgs& a, FormShared<3>& sh, int e, int tid) {
  const int* conn = a.conn + (size_t)e * 8;
  if (a.prim) {
    if (tid < 96) {
      sh.F[tid] = a.prim[(size_t)conn[tid / kHexNodeLd] * kPrimLd + tid % kHexNodeLd];
    } else if (tid < 120) {
      sh.x[(tid - 96) / 3][tid % 3] = a.x[(size_t)conn[(tid - 96) / 3] * 3 + tid % 3];
    } else if (tid < 124) {
      sh.s[tid - 120] = a.s_out[(size_t)e * 4 + tid - 120];
    }
  } else if (tid < 8) {
    double f[kPrimLd];
    node_record<3>(a.gas, a.U + (size_t)conn[tid] * 5, a.x + (size_t)conn[tid] * 3, f);
    for (int k = 0; k < kHexNodeLd; k++) sh.F[tid * kHexNodeLd + k] = f[k];
    for (int k = 0; k < 3; k++) sh.x[tid][k] = a.x[(size_t)conn[tid] * 3 + k];
    sh.Mn[tid] = f[kPrimMach];
    sh.Ren[tid] = f[kPrimRe];
  }
  if (tid == 124) {
    int nf = 0;
    for (int f = 0; f < 6; f++) {
      const int c = a.bc[(size_t)e * 6 + f];
      if (c != 0 && c < 100) {  // FDVGalerkin.h:460
        sh.faces[nf] = f;
        sh.codes[nf] = c;
        nf++;
      }
    }
    sh.nfaces = nf;
    sh.hnm = a.hnm_idx ? a.hnm_idx[e] : -1;
    sh.mask = a.rowmask ? a.rowmask[e] : 0ull;
    sh.dt = a.dt_dev ? *a.dt_dev : a.dt;
    sh.dtsq_2 = a.dt_dev ? sh.dt * sh.dt / 2.0 : a.dtsq_2;
  }
  if (tid == 96) sh.reinv = 1.0 / a.gas.creyn;
  if (tid == 97) sh.rCv = 1.0 / a.gas.Cv;
  if (tid < 104) sh.delta[tid] = (tid % 4 == 0 && (tid / 4) % 6 == 0) ? 1.0 : 0.0;
  if (tid < 64) {
    const int q = tid >> 3, N = tid & 7;
    const int hi = a.hnm_idx ? a.hnm_idx[e] : -1;
    if (hi < 0) {  // shape_fn<3> for one node
      const double zx = a.gz[q >> 2], zy = a.gz[(q >> 1) & 1], zz = a.gz[q & 1];
      const double sx = ((N & 1) ^ ((N >> 1) & 1)) ? 1.0 : -1.0, sy = ((N >> 1) & 1) ? 1.0 : -1.0,
                   sz = (N >> 2) ? 1.0 : -1.0;
      const double fx = 1 + sx * zx, fy = 1 + sy * zy, fz = 1 + sz * zz;
      double* c = &sh.cM[q][4 * N];
      c[0] = 0.125 * fx * fy * fz;
      c[1] = (sx * 0.125) * fy * fz;
      c[2] = (sy * 0.125) * fx * fz;
      c[3] = (sz * 0.125) * fx * fy;
    } else if (N == 0) {
      double z[3], Phi[8], dPxi[8][3];
      gp_point<3>(a, q, z);
      shape_fn<3>(z, Phi, dPxi);
      hnm_shape<3>(a.hnm + (size_t)hi * 64, Phi, dPxi);
      for (int M = 0; M < 8; M++) {
        sh.cM[q][4 * M] = Phi[M];
        for (int j = 0; j < 3; j++) sh.cM[q][4 * M + 1 + j] = dPxi[M][j];
      }
    }
  }
}

// isoparametric Jacobian entries (q, i, k); without node records, FDV parameters (two threads)
CFDV_HD CFDV_INLINE void hex_geom_jac(const FormArgs& a, FormShared<3>& sh, int tid) {
  if (tid < 72) {
    const int q = tid / 9, ik = tid % 9, i = ik / 3, k = ik % 3;
    double j = 0.0;
#pragma unroll
    for (int N = 0; N < 8; N++) j = RN_ADD(j, RN_MUL(sh.cM[q][4 * N + 1 + k], sh.x[N][i]));
    sh.jac[q][ik] = j;
  }
  if (!a.prim && tid >= 126) fdv_pair<8>(tid == 127 ? sh.Ren : sh.Mn, tid - 126, sh.s);
}

// physical derivatives (q, N): every thread of a point inverts the point's Jacobian itself
CFDV_HD CFDV_INLINE void hex_dphi(const FormArgs& a, FormShared<3>& sh, int tid) {
  if (tid < 64) {
    const int q = tid >> 3, N = tid & 7;
    double jac[3][3], inv[3][3], d[3];
#pragma unroll
    for (int k = 0; k < 9; k++) jac[k / 3][k % 3] = sh.jac[q][k];
    const double J = geom_det<3>(jac, inv), iJ = RN_DIV(1.0, J);
    double* c = &sh.cM[q][4 * N];
    geom_dphi<3>(c + 1, jac, inv, iJ, d);
    for (int j = 0; j < 3; j++) c[1 + j] = d[j];
    if (N == 0) {
      double z[3];
      sh.wJ[q] = gp_point<3>(a, q, z) * J;
    }
  }
}

// state sums sum_N cM(q, N, t) field(N) (FDVGalerkin.h:761-797): thread (q, t, field group) keeps
// three sums, or the last two, and places them in the point's GpState, S and raw.  Summed in the
// reference's node order without contraction: on a uniform stream the gradients are rounding
// noise of terms that cancel, and the rhs there is held to the reference's own noise.
template <bool FACE>
CFDV_HD CFDV_INLINE void hex_state(FormShared<3>& sh, int lf, int tid) {
  const int q = tid >> 4, t = (tid >> 2) & 3, f0 = 3 * (tid & 3);
  if (FACE && q >= 4) return;
  const int fc = FACE ? sh.faces[lf] : 0;
  double c[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int m = 0; m < (FACE ? 4 : 8); m++) {
    const int N = FACE ? face_node(3, fc, m) : m;
    const double w = sh.cM[q][4 * N + t];
    const double* f = sh.F + N * kHexNodeLd + f0;
#pragma unroll
    for (int j = 0; j < 3; j++) c[j] = RN_ADD(c[j], RN_MUL(w, f[j]));
  }
  HexGp& g = hex_gp<FACE>(sh, q);
  double* st = reinterpret_cast<double*>(&g.st);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int f = f0 + j;
    const double v = c[j];
    if (t == 0) {
      if (f < 7) st[f] = v;             // E, T, U
      else if (f < 10) st[15 + f] = v;  // v
    } else {
      if (f == 1) st[33 + t] = v;                               // dT
      else if (f >= 2 && f < 7) st[6 + 3 * (f - 2) + t] = v;    // dU
      else if (f >= 7 && f < 10) st[24 + 3 * (f - 7) + t] = v;  // dV
    }
    if (f >= 7 && f < 10) g.raw[t][f - 7] = v;
    if (f == 10) g.S[t] = v;
  }
}

// the scalars of a point's (edited) state that the Jacobian rows share
CFDV_HD CFDV_INLINE void hex_gp_scalars(HexGp& g) {
  const GpState& f = g.st;
  const double irho = 1.0 / f.U[0];
  g.irho = irho;
  for (int k = 0; k < 3; k++) g.w[k] = f.U[1 + k] * irho;
  g.divm = f.dU[1][0] + f.dU[2][1] + f.dU[3][2];
  g.vgr = f.v[0] * f.dU[0][0] + f.v[1] * f.dU[0][1] + f.v[2] * f.dU[0][2];
  g.q2 = f.v[0] * f.v[0] + f.v[1] * f.v[1] + f.v[2] * f.v[2];
}

// domain: viscosity, conductivity, stress (lanes 0-2 of a point: one row each), shared scalars
CFDV_HD CFDV_INLINE void hex_gp_domain(const FormArgs& a, FormShared<3>& sh, int tid) {
  if (tid >= 32) return;
  const int i = tid & 3;
  HexGp& g = sh.gp[tid >> 2];
  GpState& f = g.st;
  if (i == 3) {
    hex_gp_scalars(g);
    return;
  }
  const double mu = gas_mu(a.gas, f.T);
  const double vkk = RN_ADD(RN_ADD(f.dV[0][0], f.dV[1][1]), f.dV[2][2]);
#pragma unroll
  for (int j = 0; j < 3; j++) {
    double t = RN_MUL(mu, RN_ADD(f.dV[i][j], f.dV[j][i]));
    if (i == j) t = RN_SUB(t, RN_MUL(RN_MUL(2.0 / 3.0, mu), vkk));
    f.tau[i][j] = t;
  }
  if (i == 0) {
    f.mu = mu;
    f.k = gas_k(a.gas, mu);
  }
}

// face: viscosity and conductivity, stress zero, then the boundary edits (eval2dboundary.h)
CFDV_HD CFDV_INLINE void hex_gp_face(const FormArgs& a, FormShared<3>& sh, int lf, int tid) {
  if (tid >= 4) return;
  HexGp& g = hex_gp<true>(sh, tid);
  GpState& f = g.st;
  f.mu = gas_mu(a.gas, f.T);
  f.k = gas_k(a.gas, f.mu);
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) f.tau[i][j] = 0;
  edit_face_state_3d(sh.codes[lf], f, sh.en[tid], a.gas.adiabatic);
  hex_gp_scalars(g);
}

// convective flux of node b, entry (i, r), for the optional 3D convective rhs flux
CFDV_HD CFDV_INLINE double hex_node_conv(const FormShared<3>& sh, int b, int i, int r) {
  const double* f = sh.F + b * kHexNodeLd;
  NodePrim n;
  for (int k = 0; k < 5; k++) n.U[k] = f[2 + k];
  n.p = f[11];
  return node_conv_flux_entry<3>(n, i, r);
}

// Jacobian rows: threads (r, q, i) for r = 1..4 form row r of a_i and b_i (NavierStokes3D.h:74-343
// for a general direction) and store X, A, D; row 0 (a_i(0, 1+i) = 1 alone) goes with row 1.
// The last warp tabulates the c values and divF(s) = sum_b sum_i dPhi_b,i FG_b(i, s).
template <bool FACE>
CFDV_HD CFDV_INLINE void hex_rows(const FormArgs& a, FormShared<3>& sh, int tid) {
  constexpr int NQ = FACE ? 4 : 8, NT = 3 * NQ;
  const double dt = sh.dt, h2 = sh.dtsq_2, s1 = sh.s[0], s2 = sh.s[1], s3 = sh.s[2], s4 = sh.s[3];
  const double reinv = sh.reinv;
  if (tid < 4 * NT) {
    const int r = 1 + tid / NT, q = (tid % NT) / 3, i = tid % 3;
    HexGp& g = hex_gp<FACE>(sh, q);
    const GpState& f = g.st;
    const double g1 = a.gas.gamm1;
    const double u = f.v[i], rho_i = f.dU[0][i];
    const double irho = g.irho, muD = f.mu * irho * irho * reinv, laD = -2.0 / 3.0 * muD;
    double av[5], bv[5];
    if (r < 4) {
      const int k = r - 1;
      const double vk = f.v[k], rho_k = f.dU[0][k];
      const bool d = i == k;
      av[0] = -u * vk + (d ? a.gas.gm1d2 * g.q2 : 0.0);
      bv[0] = muD * (f.dU[1 + k][i] + f.dU[1 + i][k] - 2.0 * (vk * rho_i + u * rho_k)) +
              (d ? laD * (g.divm - 2.0 * g.vgr) : 0.0);
#pragma unroll
      for (int l = 0; l < 3; l++) {
        av[1 + l] = (k == l ? u : 0.0) + (i == l ? vk : 0.0) - (d ? g1 * f.v[l] : 0.0);
        bv[1 + l] = muD * ((k == l ? rho_i : 0.0) + (i == l ? rho_k : 0.0)) + (d ? laD * f.dU[0][l] : 0.0);
      }
      av[4] = d ? g1 : 0.0;
      bv[4] = 0.0;
    } else {
      const double E = f.E, gE = a.gas.gamma * E, T1 = f.k * irho * irho * sh.rCv;
      double vm = 0.0, mv = 0.0, wt = 0.0;  // v.d_i m, v.grad m_i, w.tau_i
#pragma unroll
      for (int k = 0; k < 3; k++) {
        vm += f.v[k] * f.dU[1 + k][i];
        mv += f.v[k] * f.dU[1 + i][k];
        wt += g.w[k] * f.tau[i][k];
      }
      av[0] = u * (g1 * g.q2 - gE);
      bv[0] = muD * (vm + mv - 2.0 * (g.q2 * rho_i + u * g.vgr)) + laD * u * (g.divm - 2.0 * g.vgr) +
              reinv * (irho * wt - T1 * (-f.dU[4][i] + (2.0 * E - 3.0 * g.q2) * rho_i + 2.0 * vm));
#pragma unroll
      for (int l = 0; l < 3; l++) {
        const double vl = f.v[l];
        av[1 + l] = (i == l ? gE - a.gas.gm1d2 * g.q2 : 0.0) - g1 * u * vl;
        bv[1 + l] = muD * (vl * rho_i + (i == l ? g.vgr : 0.0)) + laD * u * f.dU[0][l] -
                    reinv * (f.tau[i][l] * irho + T1 * (2.0 * vl * rho_i - f.dU[1 + l][i]));
      }
      av[4] = a.gas.gamma * u;
      bv[4] = reinv * T1 * rho_i;
    }
    double* Tq = sh.T[q];
#pragma unroll
    for (int s = 0; s < 5; s++) {
      g.A[5 * i + r][s] = h2 * (av[s] + bv[s]);
      g.D[r - 1][5 * i + s] = s2 * av[s] + s4 * bv[s];
      Tq[(5 * r + s) * 12 + i] = -dt * (s1 * av[s] + s3 * bv[s]);
    }
    if (r == 1) {
#pragma unroll
      for (int s = 0; s < 5; s++) {
        g.A[5 * i][s] = s == 1 + i ? h2 : 0.0;
        Tq[s * 12 + i] = s == 1 + i ? -dt * s1 : 0.0;
      }
    }
  } else if (tid >= 96) {
    const int q = (tid - 96) >> 2, p = tid & 3;
    if (FACE && q >= 4) return;
    HexGp& g = hex_gp<FACE>(sh, q);
    const GpState& f = g.st;
    const double sc = -dt * s3 * reinv * g.irho;
    const double M = sc * f.mu, L = -2.0 / 3.0 * M, K = sc * f.k * sh.rCv;
    const double* w = g.w;
    const double W2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
    double dF = 0.0;
    if (p < 3) {
      const double wp = w[p], ww = (p < 2) ? w[0] * w[1 + p] : w[1] * w[2];
      g.ctab[HC_MRW + p] = (2.0 * M + L) * wp;
      g.ctab[HC_MW + p] = M * wp;
      g.ctab[HC_LW + p] = L * wp;
      g.ctab[HC_KMRW + p] = (K - (2.0 * M + L)) * wp;
      g.ctab[HC_KMW + p] = (K - M) * wp;
      g.ctab[HC_NMW + p] = -M * wp;
      g.ctab[HC_NLW + p] = -L * wp;
      g.ctab[HC_EE + p] = M * (W2 + wp * wp) + L * wp * wp - K * (W2 - f.U[4] * g.irho);
      g.ctab[HC_WW + p] = (M + L) * ww;
#pragma unroll
      for (int i = 0; i < 3; i++) dF -= f.tau[i][p] * g.S[1 + i];
    } else {
      g.ctab[HC_NMR] = -(2.0 * M + L);
      g.ctab[HC_NM] = -M;
      g.ctab[HC_NL] = -L;
      g.ctab[HC_NK] = -K;
      g.ctab[HC_ZERO] = 0.0;
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) dF -= f.tau[i][j] * g.raw[1 + i][j];
        dF -= f.k * f.dT[i] * g.S[1 + i];
      }
    }
    dF *= reinv;
    if (p == 0) g.divF[0] = 0.0;
    if (a.physical_3d_flux) {
      double d0 = 0.0;
      for (int b = 0; b < 8; b++)
        for (int i = 0; i < 3; i++) {
          const double dp = sh.cM[q][4 * b + 1 + i];
          dF += dp * hex_node_conv(sh, b, i, 1 + p);
          if (p == 0) d0 += dp * hex_node_conv(sh, b, i, 0);
        }
      if (p == 0) g.divF[0] = d0;
    }
    g.divF[1 + p] = dF;
  }
}

// h_ij of the points (a warp per point at a time) and the rhs coefficients P(i, r)
template <bool FACE>
CFDV_HD CFDV_INLINE void hex_hmat(const FormArgs& a, FormShared<3>& sh, int tid) {
  constexpr int NQ = FACE ? 4 : 8;
  const int lane = tid & 31;
  const double s2h = sh.s[1];
#if defined(__CUDACC__) && !defined(__CUDA_ARCH__)
  const unsigned long long slots = 0;  // never run on the host in a CUDA build
#else
  const unsigned long long slots = kHexCTable.v[lane];
#endif
  // this lane's entries: rows 8 mt + lane / 4, columns 8 nt + 2 (lane % 4) + e (of 15 each); the
  // column's part of T's index and whether row 0 of D_j (s2 at s = 1 + j alone) reaches it
  int tcol[2][2];
  double sd[2][2];
#pragma unroll
  for (int nt = 0; nt < 2; nt++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int col = 8 * nt + 2 * (lane & 3) + e, j = col / 5, s = col % 5;
      tcol[nt][e] = 12 * s + 3 + 3 * j;
      sd[nt][e] = s == 1 + j ? s2h : 0.0;
    }
  const bool last = (lane & 3) == 3;  // column 15 is not one
#pragma unroll 1
  for (int q = tid >> 5; q < NQ; q += 4) {
    HexGp& g = hex_gp<FACE>(sh, q);
    double* Tq = sh.T[q];
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
      const int row = 8 * mt + (lane >> 2);
      const int trow = 60 * (row % 5) + row / 5;
      const double a0 = g.A[row][0];
      double c[2][2];
#pragma unroll
      for (int nt = 0; nt < 2; nt++) {
#pragma unroll
        for (int e = 0; e < 2; e++)
          c[nt][e] = g.ctab[(slots >> (8 * (4 * mt + 2 * nt + e))) & 31u] + sd[nt][e] * a0;
        mma_f64(lane, [&](int rw, int k) { return g.A[8 * mt + rw][1 + k]; },
                [&](int k, int cl) { return g.D[k][8 * nt + cl]; }, c[nt][0], c[nt][1]);
      }
      if (row < 15) {
        double* t = Tq + trow;
        t[tcol[0][0]] = c[0][0];
        t[tcol[0][1]] = c[0][1];
        t[tcol[1][0]] = c[1][0];
        if (!last) t[tcol[1][1]] = c[1][1];
      }
    }
  }
  if (tid < 15 * NQ) {
    const int q = tid / 15, ir = tid % 15, i = ir / 5, r = ir % 5;
    const HexGp& g = hex_gp<FACE>(sh, q);
    const GpState& f = g.st;
    double fb = 0.0;
    if (r == 4) {
#pragma unroll
      for (int j = 0; j < 3; j++) fb -= f.tau[i][j] * g.raw[0][j];
      fb -= f.k * f.dT[i] * g.S[0];
    } else if (r > 0) {
      fb = -f.tau[i][r - 1] * g.S[0];
    }
    fb *= sh.reinv;
    if (a.physical_3d_flux)
      for (int b = 0; b < 8; b++) fb += sh.cM[q][4 * b] * hex_node_conv(sh, b, i, r);
    double u = 0.0;
#pragma unroll
    for (int s = 0; s < 5; s++) u += g.A[ir][s] * g.divF[s];
    sh.P[q][ir] = sh.dt * fb - u;
  }
}

// contraction: warp w owns the (r, s) entries rs0 .. rs0 + 7 (8, 6, 6 and 5 of the 25), all 64
// (N, M) pairs each; the last warp also contracts the rhs
template <bool FACE>
CFDV_HD CFDV_INLINE void hex_contract(FormShared<3>& sh, int tid) {
  constexpr int NQ = FACE ? 4 : 8;
  const int w = tid >> 5, lane = tid & 31, N = lane >> 2, M0 = 2 * (lane & 3);
  const int rs0 = w == 0 ? 0 : 2 + 6 * w, nrs = w == 0 ? 8 : (w == 3 ? 5 : 6);
  double acc[8][2], ar[2] = {0.0, 0.0};
#pragma unroll
  for (int p = 0; p < 8; p++) {
    const int rs = rs0 + p, at = (M0 * 5 + rs % 5) * kHexTileLd + N * 5 + rs / 5;
    acc[p][0] = (FACE && p < nrs) ? sh.Rt[at] : 0.0;
    acc[p][1] = (FACE && p < nrs) ? sh.Rt[at + 5 * kHexTileLd] : 0.0;
  }
#ifdef __CUDA_ARCH__
  // the G operand of pair p at this lane: row k of column (c, e): T for k > 0, the delta table for
  // k = 0, stepping by the pair and by the point (entry 25 is the row of room: its tile is unused)
  const int kk = lane & 3, c4 = N >> 1, e4 = N & 1;
  const double* tp = kk ? sh.T[0] + (rs0 + e4) * 12 + 3 * c4 + kk - 1 : sh.delta + (rs0 + e4) * 4 + c4;
  const int dp = kk ? 24 : 8, dq = kk ? kHexTLd : 0;
  const double *t0 = tp, *t1 = tp + dp, *t2 = tp + 2 * dp, *t3 = nrs == 8 ? tp + 3 * dp : tp;
#endif
#pragma unroll 1
  for (int q = 0; q < NQ; q++) {
    const double* cq = sh.cM[q];
    auto A1 = [&](int row, int k) -> double {
      if (FACE) return k == 0 ? 0.0 : -(cq[4 * row] * sh.en[q][k - 1]);
      return sh.wJ[q] * cq[4 * row + k];
    };
    auto B2 = [&](int k, int col) -> double { return cq[4 * col + k]; };
    auto PB = [&](int k, int col) -> double { return (k > 0 && col < 5) ? sh.P[q][5 * (k - 1) + col] : 0.0; };
#ifdef __CUDA_ARCH__
    const double b2 = B2(lane & 3, N), a1 = FACE ? A1(N, lane & 3) : sh.wJ[q] * b2;
    auto rd_a = [&](int, int) { return a1; };
    auto rd_b = [&](int, int) { return b2; };
    const double tv[4] = {*t0, *t1, *t2, *t3};
    t0 += dq;
    t1 += dq;
    t2 += dq;
    t3 += dq;
#pragma unroll
    for (int p = 0; p < 4; p++) {
      if (2 * p >= nrs) break;
      double g[2];
      mma_f64_fresh(lane, rd_a, [&](int, int) { return tv[p]; }, g[0], g[1]);
#pragma unroll
      for (int e = 0; e < 2; e++)
        mma_f64(lane, [&](int, int) { return g[e]; }, rd_b, acc[2 * p + e][0], acc[2 * p + e][1]);
    }
    if (w == 3) mma_f64(lane, rd_a, PB, ar[0], ar[1]);
#else
    const double* Tq = sh.T[q];
    for (int p = 0; 2 * p < nrs; p++)
      for (int e = 0; e < 2; e++) {
        const int rs = rs0 + 2 * p + e;
        auto rd_g = [&](int row, int c) {
          double v = A1(row, 0) * sh.delta[4 * rs + c];
          for (int k = 1; k < 4; k++) v += A1(row, k) * (rs < 25 ? Tq[rs * 12 + 3 * c + k - 1] : 0.0);
          return v;
        };
        mma_f64(lane, rd_g, B2, acc[2 * p + e][0], acc[2 * p + e][1]);
      }
    if (w == 3) mma_f64(lane, A1, PB, ar[0], ar[1]);
#endif
  }
#pragma unroll
  for (int p = 0; p < 8; p++)
    if (p < nrs) {
      const int rs = rs0 + p, at = (M0 * 5 + rs % 5) * kHexTileLd + N * 5 + rs / 5;
      sh.Rt[at] = acc[p][0];
      sh.Rt[at + 5 * kHexTileLd] = acc[p][1];
    }
  if (w == 3)
#pragma unroll
    for (int e = 0; e < 2; e++)
      if (M0 + e < 5) sh.rhs[N * 5 + M0 + e] = (FACE ? sh.rhs[N * 5 + M0 + e] : 0.0) + ar[e];
}

// face geometry (calc_TF_norm3D.h:9-167), one thread per face point: coefficient rows in the
// element's node numbering (zero off the face) and the weighted normal
CFDV_HD CFDV_INLINE void hex_face_geom(const FormArgs& a, FormShared<3>& sh, int lf, int q) {
  if (q >= 4) return;
  const int f = sh.faces[lf];
  const double* xf[4];
  for (int i = 0; i < 4; i++) xf[i] = sh.x[face_node(3, f, i)];
  double xl[4][3];
  const double* H = sh.hnm >= 0 ? a.hnm + (size_t)sh.hnm * 64 : nullptr;
  if (H) {
    const double* xe[8];
    for (int M = 0; M < 8; M++) xe[M] = sh.x[M];
    hnm_face_nodes_3d(H, xe, f, xl);
    for (int i = 0; i < 4; i++) xf[i] = xl[i];
  }
  double phib[4], dpidx[4][3];
  face_point_geom<3>(a.gz, a.gw, xf, q, phib, dpidx, sh.en[q]);
  if (H) hnm_face_phi_3d(H, f, phib);
  for (int k = 0; k < 32; k++) sh.cM[q][k] = 0.0;
  for (int m = 0; m < 4; m++) {
    double* c = &sh.cM[q][4 * face_node(3, f, m)];
    c[0] = phib[m];
    for (int j = 0; j < 3; j++) c[1 + j] = dpidx[m][j];
  }
}

// ApplyBC (rows of Dirichlet DOFs: zero, diagonal 0.5, rhs 0) and the store, two rows a thread
CFDV_HD CFDV_INLINE void hex_write(const FormArgs& a, FormShared<3>& sh, int e, int tid, int* bad) {
  const uint64_t mk = sh.mask;
  const size_t base = (size_t)e * 1600;
  double nf = 0.0;  // v * 0 is NaN for an entry that is not finite, and stays
  if (tid < 120) {  // rows I, I + 1 of columns tid / 20, + 6, ...: one row pair per thread
    const int I = 2 * (tid % 20);
    const unsigned m2 = (unsigned)(mk >> I) & 3u;
    for (int J = tid / 20; J < 40; J += 6) {
      const double* t = sh.Rt + J * kHexTileLd + I;
      double v0 = t[0], v1 = t[1];
      if (m2) {
        if (m2 & 1u) v0 = I == J ? 0.5 : 0.0;
        if (m2 & 2u) v1 = I + 1 == J ? 0.5 : 0.0;
      }
      nf += v0 * 0.0 + v1 * 0.0;
      const size_t at = base + J * 40 + I;
#ifdef __CUDA_ARCH__
      if (a.R64) *reinterpret_cast<double2*>(a.R64 + at) = make_double2(v0, v1);
      if (a.R32) *reinterpret_cast<float2*>(a.R32 + at) = make_float2((float)v0, (float)v1);
#else
      if (a.R64) { a.R64[at] = v0; a.R64[at + 1] = v1; }
      if (a.R32) { a.R32[at] = (float)v0; a.R32[at + 1] = (float)v1; }
#endif
    }
  }
  if (tid < 40) {
    const double v = ((mk >> tid) & 1ull) ? 0.0 : sh.rhs[tid];
    nf += v * 0.0;
    a.rhs[(size_t)e * 40 + tid] = v;
  }
  if (nf != 0.0) *bad = 1;
  if (!a.prim && tid < 4 && a.s_out) a.s_out[(size_t)e * 4 + tid] = sh.s[tid];
}

constexpr int kHexDomainSteps = 8, kHexFaceSteps = 6;

CFDV_HD CFDV_INLINE int hex_nsteps(const FormShared<3>& sh) { return kHexDomainSteps + kHexFaceSteps * sh.nfaces + 1; }

CFDV_HD CFDV_INLINE void hex_step(int k, const FormArgs& a, FormShared<3>& sh, int e, int tid, int* bad) {
  switch (k) {
    case 0: hex_load(a, sh, e, tid); return;
    case 1: hex_geom_jac(a, sh, tid); return;
    case 2: hex_dphi(a, sh, tid); return;
    case 3: hex_state<false>(sh, 0, tid); return;
    case 4: hex_gp_domain(a, sh, tid); return;
    case 5: hex_rows<false>(a, sh, tid); return;
    case 6: hex_hmat<false>(a, sh, tid); return;
    case 7: hex_contract<false>(sh, tid); return;
    default: break;
  }
  const int f = k - kHexDomainSteps;
  if (f < kHexFaceSteps * sh.nfaces) {
    const int lf = f / kHexFaceSteps;
    switch (f % kHexFaceSteps) {
      case 0: hex_face_geom(a, sh, lf, tid); return;
      case 1: hex_state<true>(sh, lf, tid); return;
      case 2: hex_gp_face(a, sh, lf, tid); return;
      case 3: hex_rows<true>(a, sh, tid); return;
      case 4: hex_hmat<true>(a, sh, tid); return;
      default: hex_contract<true>(sh, tid); return;
    }
  }
  hex_write(a, sh, e, tid, bad);
}

}  // namespace cfdv
