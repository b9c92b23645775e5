// CUDA kernels for the per-step FDV set-up: element formation (+ ApplyBC) and the
// CFL time step.  Formation is one thread block per element running the phases of
// formation.cuh (quad4) or formation_hex.cuh (hex8); the CFL step is a minimum over the element nodes with a deterministic
// two-level reduction.
#include <cuda_runtime.h>

#include <algorithm>

#include "formation.cuh"
#include "kernels.h"

namespace cfdv {

// one 64-thread block per quad4 element (formation.cuh)
__global__ void __launch_bounds__(FormTraits<2>::THREADS, FormTraits<2>::MIN_BLOCKS) fdv_form_quad_kernel(FormArgs a) {
  __shared__ FormShared<2> sh;
  const int tid = threadIdx.x, e = blockIdx.x;
  int bad = 0;
  form_step<2>(0, a, sh, e, tid, &bad);
  __syncthreads();
  const int n = form_nsteps<2>(sh);
  for (int k = 1; k < n; k++) {
    form_step<2>(k, a, sh, e, tid, &bad);
    __syncthreads();
  }
  if (bad) atomicOr(a.status, STATUS_NONFINITE_MATRIX);
}

// one 128-thread block per hex8 element (formation_hex.cuh)
__global__ void __launch_bounds__(FormTraits<3>::THREADS, CFDV_FORM3D_BLOCKS) fdv_form_hex_kernel(FormArgs a) {
  __shared__ FormShared<3> sh;
  const int tid = threadIdx.x, e = blockIdx.x;
  int bad = 0;
  hex_load(a, sh, e, tid);
  __syncthreads();
  hex_geom_jac(a, sh, tid);
  __syncthreads();
  hex_dphi(a, sh, tid);
  __syncthreads();
  hex_state<false>(sh, 0, tid);
  __syncthreads();
  hex_gp_domain(a, sh, tid);
  __syncthreads();
  hex_rows<false>(a, sh, tid);
  __syncthreads();
  hex_hmat<false>(a, sh, tid);
  __syncthreads();
  hex_contract<false>(sh, tid);
  __syncthreads();
  const int nf = sh.nfaces;
  for (int lf = 0; lf < nf; lf++) {
    hex_face_geom(a, sh, lf, tid);
    __syncthreads();
    hex_state<true>(sh, lf, tid);
    __syncthreads();
    hex_gp_face(a, sh, lf, tid);
    __syncthreads();
    hex_rows<true>(a, sh, tid);
    __syncthreads();
    hex_hmat<true>(a, sh, tid);
    __syncthreads();
    hex_contract<true>(sh, tid);
    __syncthreads();
  }
  hex_write(a, sh, e, tid, &bad);
  if (bad) atomicOr(a.status, STATUS_NONFINITE_MATRIX);
}

// node records of the state U, one thread per node
template <int NDIM>
__global__ void __launch_bounds__(128) node_record_kernel(const double* __restrict__ U, const double* __restrict__ x,
                                                          int n_nodes, GasParams g, double* __restrict__ prim) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  double f[kPrimLd];
  node_record<NDIM>(g, U + (size_t)n * (NDIM + 2), x + (size_t)n * NDIM, f);
#pragma unroll
  for (int k = 0; k < kPrimLd; k += 2)
    *reinterpret_cast<double2*>(prim + (size_t)n * kPrimLd + k) = make_double2(f[k], f[k + 1]);
}

// s1..s4 of every element from its nodes' Mach and Reynolds numbers, one thread per element and pair
template <int NNOD>
__global__ void __launch_bounds__(128) fdv_param_kernel(const double* __restrict__ prim, const int* __restrict__ conn,
                                                        int E, double* __restrict__ s_out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, e = t >> 1, which = t & 1;
  if (e >= E) return;
  double val[NNOD], s[4];
#pragma unroll
  for (int i = 0; i < NNOD; i++) val[i] = prim[(size_t)conn[(size_t)e * NNOD + i] * kPrimLd + kPrimMach + which];
  fdv_pair<NNOD>(val, which, s);
  *reinterpret_cast<double2*>(s_out + (size_t)e * 4 + 2 * which) =
      which ? make_double2(s[2], s[3]) : make_double2(s[0], s[1]);
}

cudaError_t launch_node_records(int ndim, const double* U, const double* x, int n_nodes, const int* conn, int E,
                                const GasParams& g, double* prim, double* s_out, cudaStream_t st) {
  const int gn = (n_nodes + 127) / 128, ge = (2 * E + 127) / 128;
  if (ndim == 2) {
    node_record_kernel<2><<<gn, 128, 0, st>>>(U, x, n_nodes, g, prim);
    fdv_param_kernel<4><<<ge, 128, 0, st>>>(prim, conn, E, s_out);
  } else {
    node_record_kernel<3><<<gn, 128, 0, st>>>(U, x, n_nodes, g, prim);
    fdv_param_kernel<8><<<ge, 128, 0, st>>>(prim, conn, E, s_out);
  }
  return cudaGetLastError();
}

cudaError_t launch_form(int ndim, const FormArgs& a, cudaStream_t st) {
  if (a.n_elements <= 0) return cudaSuccess;
  const int grid = a.n_elements;
  if (ndim == 2) fdv_form_quad_kernel<<<grid, FormTraits<2>::THREADS, 0, st>>>(a);
  else fdv_form_hex_kernel<<<grid, FormTraits<3>::THREADS, 0, st>>>(a);
  return cudaGetLastError();
}

// ---- refinement marks (RefineListAdaptive.h:25-36): FDVParam's s1 from the element's node
// Mach numbers, by the same node unpack and s1 arithmetic as the formation's FDV parameters
template <int NDIM>
__global__ void refine_mark_kernel(const double* __restrict__ U, const double* __restrict__ x,
                                   const int* __restrict__ conn, int E, GasParams g, double threshold,
                                   unsigned char* marks) {
  constexpr int NNOD = (NDIM == 2) ? 4 : 8, NEQ = NDIM + 2;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x) {
    double Mn[NNOD], Ren[NNOD], s[2];
    for (int i = 0; i < NNOD; i++) {
      const int n = conn[(size_t)e * NNOD + i];
      NodePrim nd;
      node_unpack<NDIM>(g, U + (size_t)n * NEQ, x + (size_t)n * NDIM, nd);
      node_mach_re<NDIM>(g, nd, &Mn[i], &Ren[i]);
    }
    fdv_pair<NNOD>(Mn, 0, s);
    marks[e] = s[0] > threshold ? 1 : 0;
  }
}

cudaError_t launch_refine_marks(int ndim, const double* U, const double* x, const int* conn, int E, const GasParams& g,
                                double threshold, unsigned char* marks, cudaStream_t st) {
  if (E <= 0) return cudaSuccess;
  const int grid = (E + 255) / 256;
  if (ndim == 2) refine_mark_kernel<2><<<grid, 256, 0, st>>>(U, x, conn, E, g, threshold, marks);
  else refine_mark_kernel<3><<<grid, 256, 0, st>>>(U, x, conn, E, g, threshold, marks);
  return cudaGetLastError();
}

// ---- CFL (MPI_CFL.h:7-56): dt = cfl * min_e min_nodes cleng_e / (|v| + sqrt(1.4 cgas T))
template <int NDIM>
__global__ void cfl_partial_kernel(const double* __restrict__ U, const int* __restrict__ conn,
                                   const double* __restrict__ cleng, int E, GasParams g, double* partial,
                                   unsigned int* count, double cfl, double* dt_out) {
  constexpr int NNOD = (NDIM == 2) ? 4 : 8, NEQ = NDIM + 2;
  double best = 1000.0;
  // one thread per (element, node): a thread per element ran its nodes' divisions and square roots
  // one after another (2275 hexes 17 -> 7 us)
  const size_t n = (size_t)E * NNOD;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    double dxn;
    if (cfl_node_len<NDIM>(U + (size_t)conn[t] * NEQ, cleng[t / NNOD], g, &dxn) && dxn < best) best = dxn;
  }
  best = block_reduce_min(best);
  // the last block to finish takes the min over the block partials: dt = cfl * min (dt stays
  // unset when no element has a finite signal speed, as in the reference where dx_dv starts
  // at 1000); a min does not depend on the order, and the last block resets the count
  __shared__ bool last;
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = best;
    __threadfence();
    last = atomicAdd(count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double all = 1000.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) all = fmin(all, __ldcg(partial + i));
  all = block_reduce_min(all);
  if (threadIdx.x == 0) {
    dt_out[0] = (all < 1000.0) ? cfl * all : 0.0;
    *count = 0u;
  }
}

cudaError_t launch_cfl(int ndim, const double* U, const int* conn, const double* cleng, int E, const GasParams& g,
                       double cfl, double* partial, unsigned int* count, int nb, double* dt_out, cudaStream_t st) {
  nb = (int)std::max<size_t>(1, std::min<size_t>(nb, ((size_t)E * (ndim == 2 ? 4 : 8) + 255) / 256));  // a block without elements only lengthens the last one's wait
  if (ndim == 2) cfl_partial_kernel<2><<<nb, 256, 0, st>>>(U, conn, cleng, E, g, partial, count, cfl, dt_out);
  else cfl_partial_kernel<3><<<nb, 256, 0, st>>>(U, conn, cleng, E, g, partial, count, cfl, dt_out);
  return cudaGetLastError();
}

}  // namespace cfdv
