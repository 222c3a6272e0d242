// The 3D residual R2(U) and the exact first-order J.v on a 3D plan (a swept, tapered
// wing's C-H block; the reference's 3D path, src/jaxrans/numerics/residual.py:54-91,
// 273-334, on the canvas of src/jaxrans/mesh/atlas3d.py:119-210).
//
// One kernel fills the primitive canvas, ghosts included (each by its chain of conditions);
// then one thread per
// face evaluates its flux once -- MUSCL on the flow rows, HLLC or Roe with a vector
// normal, the 3D diamond face gradient, the viscous flux (with QCR2000), the SA row's
// convection and diffusion -- into a face buffer, and one thread per cell sums F_hi -
// F_lo per family and adds the SA source with |curl V|.  Templated on the scalar: `double` for R(U), `Dual` (value + tangent) for
// the J.v of the first-order residual.  Every canvas index is clamped to the canvas, the
// reference's edge padding.
#include <cstdint>

#include "linesolve3d.cuh"
#include "residual3d.cuh"

namespace jr {

// U's (and, for Dual, its tangent dU's) ghost-filled primitive canvas Q, one thread a cell: a
// cell's own state, or a ghost's by its program.  One launch in place of a canvas pass and
// two launches for each of the fill's three to twelve stages.
template <class T, int NV>
__global__ void __launch_bounds__(128, 8) k3_canvas(Plan3Dev p, const double* __restrict__ U,
                                                 const double* __restrict__ dU, T* __restrict__ Q) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const int g = p.ghost_of[c];
    if (g < 0) {
      prim_cell_n<NV>(p, U, dU, Q, c);
    } else {
      T q[NV3_MAX];
      ghost_state<NV>(p, U, dU, g, q);
#pragma unroll
      for (int v = 0; v < NV; ++v) Q[(size_t)v * n + c] = q[v];
    }
  }
}

template <class T>
static void canvas3(const Plan3Dev& p, const double* U, const double* dU, T* Q, cudaStream_t st) {
  const int blocks = (p.NI * p.NJ * p.NK + 127) / 128;
  counted3();
  if (p.nvar > 5) k3_canvas<T, 6><<<blocks, 128, 0, st>>>(p, U, dU, Q);
  else k3_canvas<T, 5><<<blocks, 128, 0, st>>>(p, U, dU, Q);
}

void launch_canvas3(const Plan3Dev& p, const double* U, double* Q, cudaStream_t st) {
  canvas3<double>(p, U, nullptr, Q, st);
}

// phase 1: every face's flux once (one thread per face of the three families)
// the diamond gradients' geometry of every face (once per plan, viscous cases)
__global__ void k3_face_geometry(Plan3Dev p, double* __restrict__ geo, int nf) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    double g[10];
    face_gradient_geometry(p, a, i, j, k, g);
    for (int q = 0; q < 10; ++q) geo[(size_t)q * nf + f] = g[q];
  }
}

// every node's mean of its eight cells' gradient variables, for the evaluation's canvas Q
template <class T, int NPHI>
__global__ void k3_node_phi(Plan3Dev p, const T* __restrict__ Q) {
  const int nn = node_count(p);
  T* nb = static_cast<T*>(p.node_buf);
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nn; e += gridDim.x * blockDim.x) {
    const int I = e / ((p.NJ + 1) * (p.NK + 1)), J = (e / (p.NK + 1)) % (p.NJ + 1), K = e % (p.NK + 1);
#pragma unroll
    for (int m = 0; m < NPHI; ++m) nb[(size_t)m * nn + e] = node_phi_m(p, Q, I, J, K, m);
  }
}

void launch_face_geometry3(const Plan3Dev& p, double* geo, cudaStream_t st) {
  const int nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  counted3();
  k3_face_geometry<<<(nf + 127) / 128, 128, 0, st>>>(p, geo, nf);
}

// (FO 1: the first-order flux, 2: second order; PART as face_flux's)
template <class T, bool VISC, bool SA, int FO, int PART>
__global__ void __launch_bounds__(128) k3_face_flux(Plan3Dev p, const T* __restrict__ Q, int nf) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x)
    store_face_flux<T, VISC, SA, FO, PART>(p, Q, FO == 1, f, p.face_buf, (size_t)nf);
}

// A viscous flux reads its diamond gradient's geometry from the plan (k3_face_geometry) and
// the node values from this evaluation's node pass (k3_node_phi: each node once, not once for
// each of the twelve faces round it).  A dual-number flux goes in two launches (inviscid, then
// viscous added): each holds half the live values of the whole, so neither spills.  A flux of
// plain doubles fits in one once its gradient takes one reciprocal for its nine quotients
// (490k cells, SA, second order: 267 us for 245 + 144 us as two; the dual's viscous part
// 567 -> 390 us by the reciprocal alone).  Bound by FP64 issue and by the latency of the
// scattered node and cell loads.
template <class T, bool VISC, bool SA, int FO>
static void face_parts(const Plan3Dev& p, const T* A, int nf, cudaStream_t st) {
  const int fblocks = (nf + 127) / 128;
  if constexpr (VISC) {
    counted3(1);
    const int nn = node_count(p);
    k3_node_phi<T, SA ? 5 : 4><<<(nn + 127) / 128, 128, 0, st>>>(p, A);
    if constexpr (sizeof(T) == sizeof(double)) {
      k3_face_flux<T, VISC, SA, FO, 0><<<fblocks, 128, 0, st>>>(p, A, nf);
    } else {
      counted3(1);
      k3_face_flux<T, VISC, SA, FO, 1><<<fblocks, 128, 0, st>>>(p, A, nf);
      k3_face_flux<T, VISC, SA, FO, 2><<<fblocks, 128, 0, st>>>(p, A, nf);
    }
  } else {
    k3_face_flux<T, VISC, SA, FO, 0><<<fblocks, 128, 0, st>>>(p, A, nf);
  }
}

template <class T, bool VISC, bool SA>
static void face_phase(const Plan3Dev& p, const T* A, bool first_order, int nf, cudaStream_t st) {
  if constexpr (sizeof(T) == sizeof(double)) {
    if (!first_order) return face_parts<T, VISC, SA, 2>(p, A, nf, st);
  }
  face_parts<T, VISC, SA, 1>(p, A, nf, st);   // (the tangent is the first-order flux's)
}

// phase 2: each cell's sum of its faces' fluxes (and the SA source)
template <class T, bool SA>
__global__ void __launch_bounds__(128) k3_cell_sum(Plan3Dev p, const T* __restrict__ Q, const double* __restrict__ U,
                                                   const double* __restrict__ dU, double* __restrict__ R, int nf) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    residual_cell_from_faces<T, SA>(p, Q, p.face_buf, (size_t)nf, U, dU, R, c);
}

// ---- launchers
template <class T>
static void residual3_t(const Plan3Dev& p, const double* U, const double* dU, double* R, T* A, bool first_order,
                        cudaStream_t st) {
  const int n = p.NI * p.NJ * p.NK;
  const int blocks = (n + 127) / 128;
  canvas3<T>(p, U, dU, A, st);
  const bool visc = p.P.mu_inf > 0.0, sa = p.nvar > 5;
  const int nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  counted3(2);   // the face phase and the cell phase
  if (sa)
    face_phase<T, true, true>(p, A, first_order, nf, st);
  else if (visc)
    face_phase<T, true, false>(p, A, first_order, nf, st);
  else
    face_phase<T, false, false>(p, A, first_order, nf, st);
  if (sa)
    k3_cell_sum<T, true><<<blocks, 128, 0, st>>>(p, A, U, dU, R, nf);
  else
    k3_cell_sum<T, false><<<blocks, 128, 0, st>>>(p, A, U, dU, R, nf);
}

__global__ void k3_wall_loads(Plan3Dev p, const double* __restrict__ Q, double* __restrict__ loads) {
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < p.n_walls; w += gridDim.x * blockDim.x)
    wall_load(p, Q, w, loads + (size_t)7 * w);
}

// the loads on every wall face (7 each) at U: the primitive canvas ghost-filled first
void launch_wall_loads3(const Plan3Dev& p, const double* U, double* loads, void* A, cudaStream_t st) {
  counted3(p.n_walls > 0);
  canvas3<double>(p, U, nullptr, (double*)A, st);
  if (p.n_walls > 0) k3_wall_loads<<<(p.n_walls + 127) / 128, 128, 0, st>>>(p, (const double*)A, loads);
}

void launch_nodes3(const Plan3Dev& p, const double* Q, cudaStream_t st) {
  const int nn = node_count(p);
  counted3();
  if (p.nvar > 5) k3_node_phi<double, 5><<<(nn + 127) / 128, 128, 0, st>>>(p, Q);
  else k3_node_phi<double, 4><<<(nn + 127) / 128, 128, 0, st>>>(p, Q);
}

void launch_residual3(const Plan3Dev& p, const double* U, double* R, void* A, bool first_order, cudaStream_t st) {
  residual3_t<double>(p, U, nullptr, R, (double*)A, first_order, st);
}

void launch_jvp3(const Plan3Dev& p, const double* U, const double* v, double* Jv, void* A, cudaStream_t st) {
  residual3_t<Dual>(p, U, v, Jv, (Dual*)A, true, st);
}

}  // namespace jr
