// The linearised 3D J.v: the bodies of its kernels (linearize3d.cu), host-and-device code.
//
// A Newton step applies one tangent map, dR1/dU at its state, to every Krylov vector, as
// the reference does (jax.linearize, src/jaxrans/solvers/implicit.py:102-116).  The map is
// stored once per step by its factors:
//
//   * per live face: the first-order flux's derivatives with respect to the primitive
//     states either side (5 x 10), the SA row's upwind value and mass flux, and the
//     scalars the viscous flux's tangent needs -- the viscosities, the stress per unit
//     viscosity and the heat-flux gradient along the face, their derivatives with respect
//     to the face temperature, density, pressure and nu~, the face velocity -- with the
//     face's gradient geometry and area vector beside them;
//   * per block cell: the SA source's derivatives with respect to rho, p, nu~ and, as two
//     vectors, curl V and grad nu~.
//
// A matrix-vector product then has no division, root or power left: it maps the tangents
// of (rho, u, v, w, p, nu~, T) through these factors.
#pragma once
#include "duals.cuh"
#include "residual3d.cuh"

namespace jr {

// The factors of a face, by number; a chunk of LIN_K faces along k keeps each factor's
// LIN_K values together (64 bytes, two sectors), the chunk's factors one after another.
constexpr int LIN_K = 8;
template <bool VISC, bool SA> struct Lin3 {
  static constexpr int A = 0;                       // d F_r / d q_s at r * 10 + s (s < 5: the low cell's)
  static constexpr int UP = 50, MASS = 51;          // SA: the upwind nu~ and the mass flux
  static constexpr int V = SA ? 52 : 50;
  static constexpr int MU = V, K = V + 1, L = V + 2, GT = V + 5, DMU = V + 6, VEL = V + 7;
  static constexpr int MUT = V + 10, COEF = V + 13, GN = V + 14, DCOEF = V + 15;   // SA
  static constexpr int GEO = V + (SA ? 18 : 10), S = GEO + 9;   // c23, c31, c12 over det; the area vector
  static constexpr int N = VISC ? S + 3 : 50;
  // QCR2000: the extra force and its derivatives with respect to the 9 velocity gradients
  // (d v_a / d x_b at 3 * b + a) and the eddy viscosity
  static constexpr int XF = N, XG = N + 3, XMU = N + 30;
  static constexpr int N_QCR = N + 33;
};
constexpr int LIN_CELL = 9;   // per cell: d src V / d (rho, p, nu~), then per unit (S x v)(3), (S nu~)(3)

__host__ __device__ __forceinline__ int lin_factors(const Plan3Dev& p) {
  if (p.nvar > 5) return p.P.c_cr1 != 0.0 ? Lin3<true, true>::N_QCR : Lin3<true, true>::N;
  return p.P.mu_inf > 0.0 ? Lin3<true, false>::N : Lin3<false, false>::N;
}

// chunks along k: every family's rows are (NI+1) x (NJ+1) of them, so one more face than
// cells fits along each axis
__host__ __device__ __forceinline__ int lin_chunks(const Plan3Dev& p) { return p.NK / LIN_K + 1; }
__host__ __device__ __forceinline__ size_t lin_words(const Plan3Dev& p) {
  return (size_t)3 * (p.NI + 1) * (p.NJ + 1) * lin_chunks(p) * LIN_K * lin_factors(p);
}
// factor 0 of face (i, j, k) of family a (factor c: c * LIN_K words on)
__host__ __device__ __forceinline__ size_t lin_at(const Plan3Dev& p, int nc, int a, int i, int j, int k) {
  const size_t chunk = (((size_t)a * (p.NI + 1) + i) * (p.NJ + 1) + j) * lin_chunks(p) + k / LIN_K;
  return chunk * nc * LIN_K + (k & (LIN_K - 1));
}

__host__ __device__ __forceinline__ bool face_live(const Plan3Dev& p, int a, int i, int j, int k) {
  const int li = i - (a == 0), lj = j - (a == 1), lk = k - (a == 2);
  const bool hi_in = i < p.NI && j < p.NJ && k < p.NK && p.interior[(i * p.NJ + j) * p.NK + k];
  const bool lo_in = li >= 0 && lj >= 0 && lk >= 0 && p.interior[(li * p.NJ + lj) * p.NK + lk];
  return hi_in || lo_in;
}

// The inviscid factors of a live face: NS columns of the Jacobian per evaluation of the
// flux.  Returns the mass flux.
template <int NS>
__host__ __device__ __forceinline__ double lin_inviscid(const Plan3Dev& p, const double* ql, const double* qh,
                                                        const double* s, double* __restrict__ out) {
  using D = Duals<NS>;
  double mass = 0.0;
#pragma unroll 1
  for (int s0 = 0; s0 < 10; s0 += NS) {
    D qL[5], qR[5], F[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      qL[v].v = ql[v];
      qR[v].v = qh[v];
#pragma unroll
      for (int t = 0; t < NS; ++t) {
        qL[v].d[t] = s0 + t == v ? 1.0 : 0.0;
        qR[v].d[t] = s0 + t == 5 + v ? 1.0 : 0.0;
      }
    }
    riemann3(p.P.flux, qL, qR, s, p.P.gamma, F);
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int t = 0; t < NS; ++t)
        if (s0 + t < 10) out[(size_t)(r * 10 + s0 + t) * LIN_K] = F[r].d[t];
    mass = F[0].v;
  }
  return mass;
}

// Every factor of live face (i, j, k) of family a at the ghost-filled canvas Q (and, of a
// viscous flow, the node values of Q in p.node_buf)
template <bool VISC, bool SA>
__host__ __device__ void linearize_face3(const Plan3Dev& p, const double* Q, int a, int i, int j, int k,
                                         double* __restrict__ out) {
  using X = Lin3<VISC, SA>;
  constexpr int NV = SA ? 6 : 5;
  const double g = p.P.gamma;
  double ql[NV3_MAX], qh[NV3_MAX], s[3];
  load_cell_n<NV>(p, Q, cell_index(p, i - (a == 0), j - (a == 1), k - (a == 2)), ql);
  load_cell_n<NV>(p, Q, cell_index(p, i, j, k), qh);
  face_vector(p, a, i, j, k, s);
  const double mass = lin_inviscid<2>(p, ql, qh, s, out);
  auto put = [&](int c, double x) { out[(size_t)c * LIN_K] = x; };
  if constexpr (SA) {
    put(X::UP, mass > 0.0 ? ql[5] : qh[5]);
    put(X::MASS, mass);
  }
  if constexpr (VISC) {
    double grad[3][5];
    face_gradient_stored<double, SA ? 5 : 4>(p, ql, qh, a, i, j, k, grad);
    double vel[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) vel[m] = 0.5 * (ql[1 + m] + qh[1 + m]);
    const double Tf = 0.5 * (g * ql[4] / ql[0] + g * qh[4] / qh[0]);
    const Dual mul = viscosity3(p.P, Dual{Tf, 1.0});
    double mu = mul.v, kc = mul.v / (PR_LAMINAR * (g - 1.0));
    double mut = 0.0;
    if constexpr (SA) {
      using D = Duals<3>;   // with respect to the face rho, p, nu~
      D rho{0.5 * (ql[0] + qh[0]), {1.0, 0.0, 0.0}}, pr{0.5 * (ql[4] + qh[4]), {0.0, 1.0, 0.0}};
      D nu{0.5 * (ql[5] + qh[5]), {0.0, 0.0, 1.0}};
      const D muf = viscosity3(p.P, g * pr / rho);
      const D mt = eddy_viscosity(p.P.sa, rho, nu * p.P.mu_inf, muf / rho);
      const D coef = diffusion_coefficient(p.P.sa, rho, nu * p.P.mu_inf, muf);
      mut = mt.v;
      mu = mu + mut;
      kc = kc + mut / (PR_TURBULENT * (g - 1.0));
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        put(X::MUT + t, mt.d[t]);
        put(X::DCOEF + t, coef.d[t]);
      }
      put(X::COEF, coef.v);
      put(X::GN, grad[0][4] * s[0] + grad[1][4] * s[1] + grad[2][4] * s[2]);
    }
    put(X::MU, mu);
    put(X::K, kc);
    put(X::DMU, mul.d);
    put(X::GT, grad[0][3] * s[0] + grad[1][3] * s[1] + grad[2][3] * s[2]);
    const double ttd = (2.0 / 3.0) * (grad[0][0] + grad[1][1] + grad[2][2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double l = -ttd * s[c];
#pragma unroll
      for (int d = 0; d < 3; ++d) l += (grad[d][c] + grad[c][d]) * s[d];
      put(X::L + c, l);
      put(X::VEL + c, vel[c]);
      put(X::S + c, s[c]);
    }
    const size_t nf = (size_t)face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
    const size_t f = (size_t)face_flat(p, a, i, j, k);
    const double inv = 1.0 / p.face_geo[9 * nf + f];
#pragma unroll
    for (int q = 0; q < 9; ++q) put(X::GEO + q, p.face_geo[(size_t)q * nf + f] * inv);
    if constexpr (SA) {
      if (p.P.c_cr1 != 0.0) {
        // one column per velocity gradient, then the eddy viscosity's
#pragma unroll 1
        for (int col = 0; col < 10; ++col) {
          Dual gd[3][5], extra[3][3];
          for (int b = 0; b < 3; ++b)
            for (int c = 0; c < 3; ++c) gd[b][c] = Dual{grad[b][c], col == 3 * b + c ? 1.0 : 0.0};
          qcr_extra(gd, Dual{mut, col == 9 ? 1.0 : 0.0}, p.P.c_cr1, extra);
          for (int c = 0; c < 3; ++c) {
            const Dual fx = extra[c][0] * s[0] + extra[c][1] * s[1] + extra[c][2] * s[2];
            put(col < 9 ? X::XG + 9 * c + col : X::XMU + c, fx.d);
            if (col == 0) put(X::XF + c, fx.v);
          }
        }
      }
    }
  }
}

// The SA source's factors of block cell c (LIN_CELL planes of n cells): the source times
// the volume, so that curl V and grad nu~ enter by their Green-Gauss sums, sum S x v and
// sum S nu~ over the faces, with the cell's 1 / V cancelled.
__host__ __device__ __forceinline__ void linearize_cell3(const Plan3Dev& p, const double* Q, int c,
                                                         double* __restrict__ out) {
  const int n = p.NI * p.NJ * p.NK;
  const int i = c / (p.NJ * p.NK), j = (c / p.NK) % p.NJ, k = c % p.NK;
  const Physics3& P = p.P;
  double qc[NV3_MAX], curl[3] = {0.0, 0.0, 0.0}, gn[3] = {0.0, 0.0, 0.0};
  load_cell_n<6>(p, Q, c, qc);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int o = side ? 1 : -1;
      double qn[NV3_MAX], s[3], v[3];
      load_cell_n<6>(p, Q, cell_index(p, i + (a == 0) * o, j + (a == 1) * o, k + (a == 2) * o), qn);
      face_vector(p, a, i + (a == 0) * side, j + (a == 1) * side, k + (a == 2) * side, s);
      for (int m = 0; m < 3; ++m) v[m] = 0.5 * (qc[1 + m] + qn[1 + m]) * o;
      const double nu = 0.5 * (qc[5] + qn[5]) * o;
      curl[0] += s[1] * v[2] - s[2] * v[1];
      curl[1] += s[2] * v[0] - s[0] * v[2];
      curl[2] += s[0] * v[1] - s[1] * v[0];
      for (int m = 0; m < 3; ++m) gn[m] += nu * s[m];
    }
  }
  const double vol = p.volume[c];
  const double sq = (curl[0] * curl[0] + curl[1] * curl[1]) + curl[2] * curl[2];
  const double len = sq > 0.0 ? sqrt(sq) : 0.0;
  using D = Duals<4>;   // with respect to rho, p, nu~, |curl V|
  D rho{qc[0], {1.0, 0.0, 0.0, 0.0}}, pr{qc[4], {0.0, 1.0, 0.0, 0.0}}, nu{qc[5], {0.0, 0.0, 1.0, 0.0}};
  D omega{len / vol, {0.0, 0.0, 0.0, 1.0}};
  D Pr, Dd;
  const D mu = viscosity3(P, P.gamma * pr / rho);
  sa_source(P.sa, nu * P.mu_inf, mu / rho, omega, p.distance[c], Pr, Dd);
  const double cb = P.sa.c_b2 / P.sa.sigma * P.mu_inf;
  const double gg = ((gn[0] * gn[0] + gn[1] * gn[1]) + gn[2] * gn[2]) / (vol * vol);
  const D src = rho * ((Pr - Dd) / P.mu_inf + cb * gg);
#pragma unroll
  for (int t = 0; t < 3; ++t) out[(size_t)t * n + c] = src.d[t] * vol;
  const double wc = len > 0.0 ? src.d[3] / len : 0.0, wn = 2.0 * qc[0] * cb / vol;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    out[(size_t)(3 + m) * n + c] = wc * curl[m];
    out[(size_t)(6 + m) * n + c] = wn * gn[m];
  }
}

}  // namespace jr
