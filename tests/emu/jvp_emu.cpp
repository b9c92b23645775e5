// Test-only CPU build of the JVP's warp code (cfdv_b200/csrc/adjoint_tangent.cuh): the 32 lanes
// run as the fibers of adj_emu.cpp.  Used only by tests/test_jvp_emulated.py.
#include "adj_emu.cpp"
#include "../../cfdv_b200/csrc/adjoint_tangent.cuh"

namespace {
template <int NDIM>
void jvp_lane(int lane) {
  static WarpJvpShared<NDIM> sh;
  EmuLanes L{lane, g_warp};
  for (int e0 = 0; e0 < g_args->n_elements; e0 += WarpJvp<NDIM>::EPW) warp_jvp<NDIM>(*g_args, sh, e0, lane, L);
  if (lane < 31) setcontext(&g_warp->ctx[lane + 1]);
  setcontext(&g_warp->main_ctx);
}
}  // namespace

extern "C" void emu_jvp_warp(int ndim, int n_elements, const double* U, const double* x, const int* conn,
                             const int* bc, const uint64_t* rowmask, double gamma, double M, double Re, double Pr,
                             double Tinf, double Tw, int adiabatic, double dt, int physical_3d_flux, const double* dU,
                             const double* tU, double t_dt, double t_mach, double* out) {
  FunctionalArgs a;
  std::memset(&a, 0, sizeof(a));
  a.gas = make_gas(gamma, M, Re, Pr, Tinf, Tw, adiabatic);
  a.dt = dt;
  gauss_legendre(2, a.gz, a.gw);
  a.n_elements = n_elements;
  a.physical_3d_flux = physical_3d_flux;
  a.U = U; a.x = x; a.conn = conn; a.bc = bc; a.rowmask = rowmask;
  a.hnm_idx = g_hnm_idx; a.hnm = g_hnm;
  a.dU = dU; a.tU = tU; a.t_dt = t_dt; a.t_mach = t_mach; a.out = out;
  FiberWarp w;
  g_warp = &w;
  g_args = &a;
  for (int l = 0; l < 32; l++) {
    w.count[l] = 0;
    w.stack[l].resize(1 << 20);
    getcontext(&w.ctx[l]);
    w.ctx[l].uc_stack.ss_sp = w.stack[l].data();
    w.ctx[l].uc_stack.ss_size = w.stack[l].size();
    w.ctx[l].uc_link = nullptr;
    makecontext(&w.ctx[l], (void (*)())(ndim == 2 ? jvp_lane<2> : jvp_lane<3>), 1, l);
  }
  swapcontext(&w.main_ctx, &w.ctx[0]);
}
