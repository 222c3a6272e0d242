// The 3D Newton step on the device: newton3d.cuh's driver over kernel-backed vector
// operations (the residual, J.v, wave speeds and line solve of residual3d.cu and
// linesolve3d.cu; dot products by a fixed-order two-stage reduction, so a step is
// bitwise reproducible while its products take the same of their two forms: matvec below).
// The device has its own form of the driver's GMRES cycle: the
// scalars of an Arnoldi step stay on the device (Gmres3), so its six kernels follow one
// another without a word from the host, which reads H once a cycle for the least squares.
#include <algorithm>
#include <cstdio>

#include "linesolve3d.cuh"
#include "newton3d.cuh"
#include "newton3d_ops.cuh"
#include "orth.cuh"

namespace jr {

constexpr int RED3_BLOCKS = 296, RED3_THREADS = 256;

__global__ void k3_vdt_add(size_t N, size_t n, const double* __restrict__ vdt, const double* __restrict__ z,
                           double* __restrict__ w) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x)
    w[e] = vdt[e % n] * z[e] + w[e];
}

__global__ void k3_axpy(size_t N, double al, const double* __restrict__ x, double* __restrict__ y) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x)
    y[e] = y[e] + al * x[e];
}

__global__ void k3_scale(size_t N, double al, const double* x, double* y) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x)
    y[e] = al * x[e];
}

// per block, fixed-order sums of (a_e b_e) and, for the density norm, of w R0^2 and w
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double s[RED3_THREADS];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = RED3_THREADS / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] = s[threadIdx.x] + s[threadIdx.x + o];
    __syncthreads();
  }
  const double out = s[0];
  __syncthreads();
  return out;
}

__global__ void k3_dot_partial(size_t N, const double* __restrict__ a, const double* __restrict__ b,
                               double* __restrict__ partial) {
  double acc = 0.0;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x)
    acc = acc + a[e] * b[e];
  const double t = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

// ---- CGS2 against the basis: three passes, each reading the basis once
//   0: h1 = V^T w;  1: w -= V h1, then h2 = V^T w;  2: w -= V h2, then |w| and column j of H.
// A thread holds its elements' entries of every vector in registers, so pass 1 updates w and
// takes its dots from one read of the basis (the two as separate passes read it twice).  One
// block of 256 threads an SM: NK entries of E elements (16-byte loads where N is even) and NK
// sums fill the registers, and 32 x 16 bytes a thread are what the reads need in flight.  On
// the 3.9M-cell wing (215 MB a vector) bound by HBM: pass 0 against 17 to 30 vectors reads
// 6.8 TB/s, pass 1 4.9; a step's three passes over 30 vectors 1.9 ms on average where separate
// dots (w read again for each vector) and updates took 2.8.  The two-element updates spill: 124
// bytes a thread at 16 vectors (two blocks an SM), 116 at 32.  Means over the vectors each form
// takes in a cycle of 30, passes 0 and 1: 1 to 8 vectors 9 and 7 us on a 49k-cell wing, 9 to 16
// 14 and 13, 17 to 30 22 and 27; on the 3.9M-cell wing 9 to 16 409 and 538 us, 17 to 30 844 and 1194.
// The sums are fixed by N alone.
template <int E> struct Elems {
  double x[E];
};
template <int E> __device__ __forceinline__ Elems<E> load_elems(const double* p) {
  Elems<E> r;
  if constexpr (E == 2) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    r.x[0] = t.x;
    r.x[1] = t.y;
  } else {
    r.x[0] = *p;
  }
  return r;
}
template <int E> __device__ __forceinline__ void store_elems(double* p, const Elems<E>& v) {
  if constexpr (E == 2) *reinterpret_cast<double2*>(p) = make_double2(v.x[0], v.x[1]);
  else *p = v.x[0];
}

// The dots of vectors k0 .. k0 + nk - 1 (nk <= NK) with w, after (UPDATE) w -= sum h V over
// the same vectors; hin, hout: the scalars of vector k0.
template <int NK, int E, bool UPDATE>
__global__ void __launch_bounds__(ORTH_THREADS, NK <= 16 ? 2 : 1) k3_orth_dots(size_t N, int nk, const double* __restrict__ V,
                                                                double* __restrict__ w,
                                                                const double* __restrict__ hin, double* hout,
                                                                double* partial, unsigned* ticket) {
  __shared__ double h[NK], total[NK];
  if (UPDATE) {
    if ((int)threadIdx.x < NK) h[threadIdx.x] = (int)threadIdx.x < nk ? hin[threadIdx.x] : 0.0;
    __syncthreads();
  }
  double acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = 0.0;
  const size_t step = (size_t)gridDim.x * ORTH_THREADS * E;
  for (size_t e = ((size_t)blockIdx.x * ORTH_THREADS + threadIdx.x) * E; e < N; e += step) {
    Elems<E> we = load_elems<E>(w + e), v[NK];
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk) v[k] = load_elems<E>(V + (size_t)k * N + e);
    if (UPDATE) {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NK; ++k)
          if (k < nk) s += h[k] * v[k].x[i];
        we.x[i] -= s;
      }
      store_elems<E>(w + e, we);
    }
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk)
#pragma unroll
        for (int i = 0; i < E; ++i) acc[k] += v[k].x[i] * we.x[i];
  }
  if (finish_sums<NK>(acc, partial, ticket, gridDim.x, total) && (int)threadIdx.x < nk) hout[threadIdx.x] = total[threadIdx.x];
}

// w -= sum h V over all nk vectors, and with `column` |w| and column j of H (m + 1 rows,
// row-major H[i * m + j])
template <int E>
__global__ void __launch_bounds__(ORTH_THREADS) k3_orth_update(size_t N, int nk, const double* __restrict__ V,
                                                               double* __restrict__ w, const double* __restrict__ hin,
                                                               Gmres3* g, int j, int m, int column, double* partial) {
  __shared__ double h[MAX_RESTART3 + 1], total[8];
  if ((int)threadIdx.x < nk) h[threadIdx.x] = hin[threadIdx.x];
  __syncthreads();
  double acc[8] = {};
  const size_t step = (size_t)gridDim.x * ORTH_THREADS * E;
  for (size_t e = ((size_t)blockIdx.x * ORTH_THREADS + threadIdx.x) * E; e < N; e += step) {
    Elems<E> we = load_elems<E>(w + e);
    double s[E] = {};
    for (int k0 = 0; k0 < nk; k0 += 16) {
      Elems<E> v[16];
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k0 + k < nk) v[k] = load_elems<E>(V + (size_t)(k0 + k) * N + e);
#pragma unroll
      for (int k = 0; k < 16; ++k)
        if (k0 + k < nk)
#pragma unroll
          for (int i = 0; i < E; ++i) s[i] += h[k0 + k] * v[k].x[i];
    }
#pragma unroll
    for (int i = 0; i < E; ++i) {
      we.x[i] -= s[i];
      acc[0] += we.x[i] * we.x[i];
    }
    store_elems<E>(w + e, we);
  }
  if (!column || !finish_sums<8>(acc, partial, &g->ticket, gridDim.x, total)) return;
  const double nrm = sqrt(total[0]);
  for (int i = threadIdx.x; i < nk; i += ORTH_THREADS) g->H[i * m + j] = g->h1[i] + g->h2[i];
  if (threadIdx.x == 0) {
    g->H[(j + 1) * m + j] = nrm;
    g->inv = 1.0 / fmax(nrm, 2.2250738585072014e-308);
  }
}

__global__ void k3_cycle_begin(Gmres3* g, double inv, int m) {
  for (int e = threadIdx.x; e < (m + 1) * m; e += blockDim.x) g->H[e] = 0.0;
  if (threadIdx.x == 0) g->inv = inv;
}

struct Coeffs3 {
  double y[MAX_RESTART3], hy[MAX_RESTART3 + 1];
};

// The end of a cycle: t = sum y V, action += sum (H y) V, V_m = w / |w| (one read of the basis)
__global__ void __launch_bounds__(256) k3_combine(size_t N, int m, Coeffs3 cf, const double* __restrict__ V,
                                                  const double* __restrict__ w, const Gmres3* __restrict__ g,
                                                  double* __restrict__ t, double* __restrict__ action) {
  const double inv = g->inv;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x) {
    double s = 0.0, a = action[e];
    for (int k0 = 0; k0 < m; k0 += 8) {
      double v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = k0 + k < m ? V[(size_t)(k0 + k) * N + e] : 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k0 + k < m) {
          s += cf.y[k0 + k] * v[k];
          a += cf.hy[k0 + k] * v[k];
        }
    }
    t[e] = s;
    action[e] = a + cf.hy[m] * (inv * w[e]);
  }
}

// x += z; r = b - action
__global__ void k3_cycle_end(size_t N, const double* __restrict__ z, const double* __restrict__ b,
                             const double* __restrict__ action, double* __restrict__ x, double* __restrict__ r) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x) {
    x[e] += z[e];
    r[e] = b[e] - action[e];
  }
}

// z = v = *scale src: the Arnoldi vector without a preconditioner
__global__ void k3_scale_copy(size_t N, const double* __restrict__ scale, const double* __restrict__ src,
                              double* __restrict__ v, double* __restrict__ z) {
  const double s = *scale;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < N; e += (size_t)gridDim.x * blockDim.x) {
    const double x = s * src[e];
    v[e] = x;
    z[e] = x;
  }
}

__global__ void k3_norm_partial(Plan3Dev p, const double* __restrict__ R, double* __restrict__ partial) {
  const int n = p.NI * p.NJ * p.NK;
  double a = 0.0, w = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    if (p.interior[c]) {
      a = a + p.volume[c] * R[c] * R[c];
      w = w + p.volume[c];
    }
  const double ta = block_sum(a), tw = block_sum(w);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = ta;
    partial[gridDim.x + blockIdx.x] = tw;
  }
}

// the largest relative change a cell's density, pressure or nu~ would see
__global__ void k3_worst_partial(Plan3Dev p, const double* __restrict__ U, const double* __restrict__ D,
                                 double* __restrict__ partial) {
  const int n = p.NI * p.NJ * p.NK;
  const double g = p.P.gamma;
  double worst = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    double q[NV3_MAX];
    prim_at(p, U, c, q);
    double de = D[(size_t)4 * n + c];
    for (int k = 0; k < 3; ++k) de = de - q[1 + k] * D[(size_t)(1 + k) * n + c];
    const double vv = (q[1] * q[1] + q[2] * q[2]) + q[3] * q[3];
    const double dp = (g - 1.0) * (de + 0.5 * vv * D[c]);
    worst = fmax(worst, fabs(D[c]) / q[0]);
    worst = fmax(worst, fabs(dp) / q[4]);
    if (p.nvar > 5) {
      const double nh = U[(size_t)5 * n + c] / q[0];
      const double dnh = (D[(size_t)5 * n + c] - nh * D[c]) / q[0];
      worst = fmax(worst, fabs(dnh) / fmax(fabs(nh), 1.0));
    }
  }
  __shared__ double s[RED3_THREADS];
  s[threadIdx.x] = worst;
  __syncthreads();
  for (int o = RED3_THREADS / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] = fmax(s[threadIdx.x], s[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// flag 1 where U + D is not physical or D not finite
__global__ void k3_physical(Plan3Dev p, const double* __restrict__ U, const double* __restrict__ D, int* flag) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    double u[NV3_MAX], q[NV3_MAX];
    bool finite = true;
    for (int v = 0; v < p.nvar; ++v) {
      const double d = D[(size_t)v * n + c];
      finite = finite && isfinite(d);
      u[v] = U[(size_t)v * n + c] + d;
    }
    to_prim3(u, q, p.nvar, p.P.gamma);
    const bool ok = finite && q[0] > 1e-10 && q[4] > 1e-10 && isfinite(q[0]) && isfinite(q[4]);
    if (!ok) atomicOr(flag, 1);
  }
}

static int grid_of(size_t N) {
  const size_t b = (N + 255) / 256;
  return (int)(b < 4096 ? (b > 0 ? b : 1) : 4096);
}

// ---- the operations
double DeviceOps3::host_sum(int count, int halves) {
  std::vector<double> h((size_t)count * halves);
  cudaMemcpyAsync(h.data(), partial, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  double s0 = 0.0, s1 = 0.0;
  for (int b = 0; b < count; ++b) s0 = s0 + h[b];
  if (halves > 1) {
    for (int b = 0; b < count; ++b) s1 = s1 + h[count + b];
    last_second = s1;
  }
  return s0;
}

void DeviceOps3::prepare(const double* U, double cfl) {
  launch_line_factor3(p, U, cfl, line ? factor : nullptr, vdt, st);
  // the tangent map of this step's products; its canvas (A) is the residual's too, which
  // leaves the same values there
  if (lin_face != nullptr) launch_linearize3(p, U, static_cast<double*>(A), lin_face, lin_cell, st);
}

void DeviceOps3::residual(const double* U, int out) { launch_residual3(p, U, v(out), A, false, st); }

void DeviceOps3::matvec(const double* U, double, int src, int out) {
  if (lin_face != nullptr) {
    launch_lin_jv3(p, U, static_cast<const double*>(A), lin_face, lin_cell, lin_dq, v(src), vdt, v(out), st);
    return;
  }
  launch_jvp3(p, U, v(src), v(out), A, st);
  counted3();
  k3_vdt_add<<<grid_of(N), 256, 0, st>>>(N, n, vdt, v(src), v(out));
}

// the factor of this step's (U, cfl), made in prepare
void DeviceOps3::precondition(const double*, double, int src, int dst) {
  launch_line_apply3(p, factor, v(src), v(dst), nullptr, nullptr, st);
}

template <int NK, int E>
static void orth_dots(DeviceOps3& o, bool update, int blocks, int nk, const double* V, double* w, const double* hin,
                      double* hout) {
  counted3();
  if (update)
    k3_orth_dots<NK, E, true><<<blocks, ORTH_THREADS, 0, o.st>>>(o.N, nk, V, w, hin, hout, o.partial, &o.gm->ticket);
  else
    k3_orth_dots<NK, E, false><<<blocks, ORTH_THREADS, 0, o.st>>>(o.N, nk, V, w, hin, hout, o.partial, &o.gm->ticket);
}

// orthogonalise W_ against V(0) .. V(j) and make column j of H
template <int E> static void orthogonalise(DeviceOps3& o, int j, int m) {
  const int nk = j + 1;
  const size_t per = (size_t)ORTH_THREADS * E;
  const int blocks = (int)std::min<size_t>(ORTH_BLOCKS, (o.N + per - 1) / per);
  const double* V = o.v(o.V(0));
  double* w = o.v(DeviceOps3::W_);
  Gmres3* g = o.gm;
  auto dots = [&](bool update, int k0, int count, const double* hin, double* hout) {
    const double* Vk = V + (size_t)k0 * o.N;
    // (few vectors: registers for two blocks an SM, which the reads in flight then need)
    if (count <= 8) orth_dots<8, E>(o, update, blocks * 2, count, Vk, w, hin, hout + k0);
    else if (count <= 16) orth_dots<16, E>(o, update, blocks * 2, count, Vk, w, hin, hout + k0);
    else orth_dots<ORTH_NK, E>(o, update, blocks, count, Vk, w, hin, hout + k0);
  };
  auto update = [&](const double* h, int column) {
    counted3();
    k3_orth_update<E><<<blocks * 2, ORTH_THREADS, 0, o.st>>>(o.N, nk, V, w, h, g, j, m, column, o.partial);
  };
  for (int k0 = 0; k0 < nk; k0 += ORTH_NK) dots(false, k0, std::min(ORTH_NK, nk - k0), nullptr, g->h1);
  if (nk <= ORTH_NK) {
    dots(true, 0, nk, g->h1, g->h2);
  } else {   // more vectors than a thread holds: the update, then the dots in slices
    update(g->h1, 0);
    for (int k0 = 0; k0 < nk; k0 += ORTH_NK) dots(false, k0, std::min(ORTH_NK, nk - k0), nullptr, g->h2);
  }
  update(g->h2, 1);
}

// Right-preconditioned restarted GMRES (src/jaxrans/solvers/krylov.py:34-97), an Arnoldi step's scalars
// on the device: (V/dt + J) X = B, ACTION = A X
int gmres3(DeviceOps3& ops, const double* U, double cfl, const Newton3Config& c, int B, int X, int ACTION) {
  const double tiny = 2.2250738585072014e-308;
  const double rcond = 2.220446049250313e-16 * (c.restart + 1);
  const int m = c.restart, grid = grid_of(ops.N);
  const size_t N = ops.N;
  const double bn = ops.nrm2(B);
  ops.zero(X);
  ops.copy(B, DeviceOps3::R_);
  ops.zero(ACTION);
  std::vector<double> H((size_t)(m + 1) * m), y;
  for (int k = 0; k < c.maxiter; ++k) {
    const double beta = k == 0 ? bn : ops.nrm2(DeviceOps3::R_);
    if (!(beta > c.tol * bn)) break;
    counted3();
    k3_cycle_begin<<<1, 256, 0, ops.st>>>(ops.gm, 1.0 / std::fmax(beta, tiny), m);
    for (int j = 0; j < m; ++j) {
      const double* src = ops.v(j == 0 ? DeviceOps3::R_ : DeviceOps3::W_);
      double *z = ops.v(DeviceOps3::Z_), *vj = ops.v(ops.V(j));
      if (c.preconditioner >= 1) {
        launch_line_apply3(ops.p, ops.factor, src, z, &ops.gm->inv, vj, ops.st);
      } else {
        counted3();
        k3_scale_copy<<<grid, 256, 0, ops.st>>>(N, &ops.gm->inv, src, vj, z);
      }
      ops.matvec(U, cfl, DeviceOps3::Z_, DeviceOps3::W_);
      if (N % 2 == 0) orthogonalise<2>(ops, j, m);
      else orthogonalise<1>(ops, j, m);
    }
    cudaMemcpyAsync(H.data(), ops.gm->H, H.size() * sizeof(double), cudaMemcpyDeviceToHost, ops.st);
    cudaStreamSynchronize(ops.st);
    givens_lstsq(H, m, beta, rcond, y);
    Coeffs3 cf{};
    for (int i = 0; i <= m; ++i) {
      double s = 0.0;
      for (int j = 0; j < m; ++j) s = s + H[(size_t)i * m + j] * y[j];
      cf.hy[i] = s;
      if (i < m) cf.y[i] = y[i];
    }
    counted3();
    k3_combine<<<grid, 256, 0, ops.st>>>(N, m, cf, ops.v(ops.V(0)), ops.v(DeviceOps3::W_), ops.gm,
                                         ops.v(DeviceOps3::T_), ops.v(ACTION));
    if (c.preconditioner >= 1) ops.precondition(U, cfl, DeviceOps3::T_, DeviceOps3::Z_);
    else ops.copy(DeviceOps3::T_, DeviceOps3::Z_);
    counted3();
    k3_cycle_end<<<grid, 256, 0, ops.st>>>(N, ops.v(DeviceOps3::Z_), ops.v(B), ops.v(ACTION), ops.v(X),
                                           ops.v(DeviceOps3::R_));
  }
  return 0;
}

double DeviceOps3::dot(int a, int b) {
  counted3();
  k3_dot_partial<<<RED3_BLOCKS, RED3_THREADS, 0, st>>>(N, v(a), v(b), partial);
  return host_sum(RED3_BLOCKS, 1);
}

void DeviceOps3::axpy(double al, int x, int y) {
  counted3();
  k3_axpy<<<grid_of(N), 256, 0, st>>>(N, al, v(x), v(y));
}
void DeviceOps3::scale(double al, int x, int y) {
  counted3();
  k3_scale<<<grid_of(N), 256, 0, st>>>(N, al, v(x), v(y));
}
void DeviceOps3::copy(int x, int y) { cudaMemcpyAsync(v(y), v(x), N * sizeof(double), cudaMemcpyDeviceToDevice, st); }
void DeviceOps3::zero(int y) { cudaMemsetAsync(v(y), 0, N * sizeof(double), st); }

double DeviceOps3::density_norm(int r) {
  counted3();
  k3_norm_partial<<<RED3_BLOCKS, RED3_THREADS, 0, st>>>(p, v(r), partial);
  const double a = host_sum(RED3_BLOCKS, 2);
  return sqrt(a / last_second);
}

double DeviceOps3::worst_ratio(const double* U, int du) {
  counted3();
  k3_worst_partial<<<RED3_BLOCKS, RED3_THREADS, 0, st>>>(p, U, v(du), partial);
  std::vector<double> h(RED3_BLOCKS);
  cudaMemcpyAsync(h.data(), partial, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  double w = 0.0;
  for (double x : h) w = fmax(w, x);
  return w;
}

bool DeviceOps3::physical_after(const double* U, int du) {
  cudaMemsetAsync(flag, 0, sizeof(int), st);
  counted3();
  k3_physical<<<grid_of(n), 128, 0, st>>>(p, U, v(du), flag);
  int h = 0;
  cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
  cudaStreamSynchronize(st);
  return h == 0;
}

void DeviceOps3::add_to_state(double* U, int du) {
  counted3();
  k3_axpy<<<grid_of(N), 256, 0, st>>>(N, 1.0, v(du), U);
}

size_t DeviceOps3::work_doubles(size_t N, size_t n, int m) {
  // the vectors, V/dt and the reductions' partial sums (and room to keep each 16-byte aligned)
  return (size_t)(BASE + m + 1) * N + n + 2 + std::max<size_t>((size_t)2 * RED3_BLOCKS, (size_t)4 * ORTH_BLOCKS * ORTH_NK);
}

void DeviceOps3::bind(double* work, Gmres3* scalars, int m) {
  vecs = work;
  vdt = work + (size_t)(BASE + m + 1) * N;
  partial = vdt + n;
  gm = scalars;
  flag = &scalars->flag;
}

double newton_step3_device(DeviceOps3& ops, double* U, double& cfl, double& res_prev, const Newton3Config& c) {
  return newton_step3(ops, U, cfl, res_prev, c);
}

}  // namespace jr
