// The 3D wave speeds and line preconditioner, per-face, per-cell and per-chain bodies (host
// and device code; linesolve3d.cu launches them, one thread each): the reference's
// face_wave_speeds (src/jaxrans/numerics/residual.py:169-203) and line_j
// (src/jaxrans/solvers/preconditioners.py:209-306) on a 3D plan -- 5x5 mean-flow chain
// blocks, the SA row on its own scalar chains -- solved along each chain by the block
// Thomas algorithm (src/jaxrans/core/linalg.py:80-132).
#pragma once
#include "residual3d.cuh"

namespace jr {


// primitive state of canvas cell c straight from U (no ghost fill)
__host__ __device__ __forceinline__ void prim_at(const Plan3Dev& p, const double* U, int c, double q[NV3_MAX]) {
  const int n = p.NI * p.NJ * p.NK;
  double u[NV3_MAX];
  for (int v = 0; v < p.nvar; ++v) u[v] = U[(size_t)v * n + c];
  to_prim3(u, q, p.nvar, p.P.gamma);
}

// the two cells either side of face (a, i, j, k), each replaced by its partner across a
// block face (the neighbour map), the canvas edge repeated
__host__ __device__ __forceinline__ void face_cells(const Plan3Dev& p, int a, int i, int j, int k, int& lo, int& hi) {
  int l[3] = {i, j, k}, h[3] = {i, j, k};
  l[a] -= 1;
  lo = p.neighbours[cell_index(p, l[0], l[1], l[2])];
  hi = p.neighbours[cell_index(p, h[0], h[1], h[2])];
}

// face-averaged primitive state and volume (src/jaxrans/mesh/atlas.py:169-183)
__host__ __device__ __forceinline__ void face_average(const Plan3Dev& p, const double* U, int a, int i, int j, int k,
                                                      double qf[NV3_MAX], double& vol) {
  int lo, hi;
  face_cells(p, a, i, j, k, lo, hi);
  double ql[NV3_MAX], qh[NV3_MAX];
  prim_at(p, U, lo, ql);
  prim_at(p, U, hi, qh);
  for (int v = 0; v < p.nvar; ++v) qf[v] = 0.5 * (ql[v] + qh[v]);
  vol = 0.5 * (p.volume[lo] + p.volume[hi]);
}

// lambda = |V.S| + a|S| at the face-averaged state, plus the thin-layer viscous term
__host__ __device__ __forceinline__ double wave_speed(const Plan3Dev& p, const double* U, int a, int i, int j, int k) {
  const Physics3& P = p.P;
  const double g = P.gamma;
  double qf[NV3_MAX], vol, s[3];
  face_average(p, U, a, i, j, k, qf, vol);
  face_vector(p, a, i, j, k, s);
  const double ss = (s[0] * s[0] + s[1] * s[1]) + s[2] * s[2];
  double vn = (qf[1] * s[0] + qf[2] * s[1]) + qf[3] * s[2];
  double lam = (vn >= 0.0 ? vn : -vn) + sqrt(g * qf[4] / qf[0]) * sqrt(ss);
  if (P.mu_inf > 0.0) {
    double mu = viscosity3(P, g * qf[4] / qf[0]);
    if (p.nvar > 5) mu = mu + eddy_viscosity(P.sa, qf[0], qf[5] * P.mu_inf, mu / qf[0]);
    lam = lam + 2.0 * g / PR_LAMINAR * mu * ss / (qf[0] * vol);
  }
  return lam;
}

// the SA row's coupling to a neighbour's mean flow: half the Jacobian of rho nu_hat V.S'
// with respect to its (rho, rho u, rho v, rho w, rho E) at its state qnb, S' = sign S:
// [-nu_hat vn, nu_hat S'x, nu_hat S'y, nu_hat S'z, 0]
__host__ __device__ __forceinline__ void sa_coupling_row(const double* qnb, const double* s, double sign,
                                                         double row[5]) {
  const double sx = sign * s[0], sy = sign * s[1], sz = sign * s[2];
  const double nu = qnb[5];
  const double vn = qnb[1] * sx + qnb[2] * sy + qnb[3] * sz;
  row[0] = 0.5 * (-nu * vn);
  row[1] = 0.5 * (nu * sx);
  row[2] = 0.5 * (nu * sy);
  row[3] = 0.5 * (nu * sz);
  row[4] = 0.5 * 0.0;
}

// ---- the factor and the solve, split by what can run in parallel.
// k3_line_faces makes each face's wave speed (and, SA, mass flux and diffusion) once instead
// of once from either side and again for the link, k3_line_cells each cell's diagonals,
// k3_line_factor the elimination down a chain, one thread a chain, and k3_line_apply the two
// sweeps, eight lanes a chain.

// prim_at with the variable count fixed at compile time (no local array)
template <int NV>
__host__ __device__ __forceinline__ void prim_at_n(const Plan3Dev& p, const double* U, int c, double q[NV3_MAX]) {
  const int n = p.NI * p.NJ * p.NK;
  double u[NV3_MAX];
#pragma unroll
  for (int v = 0; v < NV; ++v) u[v] = U[(size_t)v * n + c];
  to_prim3(u, q, NV, p.P.gamma);
}

// the line terms of face (a, i, j, k): lambda, and on the SA row the mass flux and diffusion
template <bool SA>
__host__ __device__ __forceinline__ void line_face_terms(const Plan3Dev& p, const double* U, int a, int i, int j, int k,
                                                         double& lam, double& m, double& d) {
  const Physics3& P = p.P;
  const double g = P.gamma;
  constexpr int NV = SA ? 6 : 5;
  double ql[NV3_MAX], qh[NV3_MAX], qf[NV3_MAX], s[3];
  const int lo = p.neighbours[cell_index(p, i - (a == 0), j - (a == 1), k - (a == 2))];
  const int hi = p.neighbours[cell_index(p, i, j, k)];
  prim_at_n<NV>(p, U, lo, ql);
  prim_at_n<NV>(p, U, hi, qh);
#pragma unroll
  for (int v = 0; v < NV; ++v) qf[v] = 0.5 * (ql[v] + qh[v]);
  const double vol = 0.5 * (p.volume[lo] + p.volume[hi]);
  face_vector(p, a, i, j, k, s);
  const double ss = (s[0] * s[0] + s[1] * s[1]) + s[2] * s[2];
  const double vn = (qf[1] * s[0] + qf[2] * s[1]) + qf[3] * s[2];
  lam = (vn >= 0.0 ? vn : -vn) + sqrt(g * qf[4] / qf[0]) * sqrt(ss);
  if (P.mu_inf > 0.0) {
    const double mul = viscosity3(P, g * qf[4] / qf[0]);
    double mu = mul;
    if constexpr (SA) {
      mu = mul + eddy_viscosity(P.sa, qf[0], qf[5] * P.mu_inf, mul / qf[0]);
      m = qf[0] * vn;
      d = diffusion_coefficient(P.sa, qf[0], qf[5] * P.mu_inf, mul) * ss / vol;
    }
    lam = lam + 2.0 * g / PR_LAMINAR * mu * ss / (qf[0] * vol);
  }
}

// The diagonals of cell c from its faces' terms: the sum of lambda, and (SA) the SA chain's
// diagonal (src/jaxrans/solvers/preconditioners.py:235-270)
template <bool SA>
__host__ __device__ __forceinline__ void line_cell_terms(const Plan3Dev& p, const double* U, const double* lam,
                                                         const double* mflux, const double* dflux, double cfl, int c,
                                                         double& sum, double& dsa) {
  const int i = c / (p.NJ * p.NK), j = (c / p.NK) % p.NJ, k = c % p.NK;
  int lo[3], hi[3];
  sum = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = face_flat(p, a, i, j, k);
    hi[a] = face_flat(p, a, i + (a == 0), j + (a == 1), k + (a == 2));
    sum = a == 0 ? lam[lo[a]] + lam[hi[a]] : sum + lam[lo[a]] + lam[hi[a]];
  }
  if constexpr (SA) {
    const Physics3& P = p.P;
    const double g = P.gamma, vol = p.volume[c];
    double q[NV3_MAX], own[NV3_MAX], diag = 0.0, curl[3] = {0.0, 0.0, 0.0};
    prim_at_n<6>(p, U, c, q);
    prim_at_n<6>(p, U, p.neighbours[c], own);   // the cell as its faces' means take it
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double ml = mflux[lo[a]], mh = mflux[hi[a]];
      const double out_hi = (mh > 0.0 ? mh : 0.0) + dflux[hi[a]], in_lo = (-ml > 0.0 ? -ml : 0.0) + dflux[lo[a]];
      diag = a == 0 ? out_hi + in_lo : diag + out_hi + in_lo;
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        const int o = side ? 1 : -1;
        double qn[NV3_MAX], s[3], v[3];
        prim_at_n<6>(p, U, p.neighbours[cell_index(p, i + (a == 0) * o, j + (a == 1) * o, k + (a == 2) * o)], qn);
        face_vector(p, a, i + (a == 0) * side, j + (a == 1) * side, k + (a == 2) * side, s);
#pragma unroll
        for (int m = 0; m < 3; ++m) v[m] = 0.5 * (own[1 + m] + qn[1 + m]) * o;
        curl[0] += s[1] * v[2] - s[2] * v[1];
        curl[1] += s[2] * v[0] - s[0] * v[2];
        curl[2] += s[0] * v[1] - s[1] * v[0];
      }
    }
    diag = diag / q[0];
    const double sq = (curl[0] * curl[0] + curl[1] * curl[1]) + curl[2] * curl[2];
    const double omega = sq > 0.0 ? sqrt(sq) / vol : 0.0;
    const double nu = viscosity3(P, g * q[4] / q[0]) / q[0], dist = p.distance[c];
    const double st = s_tilde(P.sa, omega, q[5] * P.mu_inf, nu, dist);
    const double fw = f_w(P.sa, r_of(P.sa, q[5] * P.mu_inf, st, dist));
    const double dest = q[5] > 0.0 ? 2.0 * P.sa.c_w1 * fw * P.mu_inf * q[5] / (dist * dist) : 0.0;
    dsa = diag + dest * vol + sum / cfl;
  }
}

// A = d(F . S)/dU (5x5, [row][variable]) of the conservative state whose primitives are q, in
// closed form (src/jaxrans/physics/euler.py:55-71), then 1/2 A - 1/2 lam I
__host__ __device__ __forceinline__ void coupling5_closed(const double* q, double sx, double sy, double sz, double lam,
                                                          double g, double B[5][5]) {
  const double S[3] = {sx, sy, sz};
  const double vn = (q[1] * sx + q[2] * sy) + q[3] * sz;
  const double vv = (q[1] * q[1] + q[2] * q[2]) + q[3] * q[3];
  const double phi = 0.5 * (g - 1.0) * vv, H = g / (g - 1.0) * q[4] / q[0] + 0.5 * vv;
  B[0][0] = -0.5 * lam;
  B[0][4] = 0.0;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    B[0][1 + b] = 0.5 * S[b];
    B[1 + b][0] = 0.5 * (phi * S[b] - q[1 + b] * vn);
    B[1 + b][4] = 0.5 * ((g - 1.0) * S[b]);
    B[4][1 + b] = 0.5 * (H * S[b] - (g - 1.0) * q[1 + b] * vn);
#pragma unroll
    for (int d = 0; d < 3; ++d)
      B[1 + b][1 + d] = 0.5 * (q[1 + b] * S[d] - (g - 1.0) * q[1 + d] * S[b]) + (b == d ? 0.5 * (vn - lam) : 0.0);
  }
  B[4][0] = 0.5 * ((phi - H) * vn);
  B[4][4] = 0.5 * (g * vn - lam);
}

// The factor's layout: four chains a group, eight rows a chain, fifteen words a row and
// element: word w of row a of chain ch at element k is
// F[((k * groups + ch / 4) * 15 + w) * 32 + (ch % 4) * 8 + a], so one word of a warp's 4 x 8
// rows is one aligned segment.  Rows 0 to 4, the mean flow: words 0 to 4 the lower block's
// row, 5 to 9 the inverse pivot's, 10 to 14 that of C = P upper.  Row 5, the SA chain: its
// lower scalar, inverse pivot (words 0, 1) and c (word 10).  The coupled form solves the SA
// chain from its far end down, beside the mean flow's way back: row 5 holds its upper scalar
// and inverse pivot in words 10, 11 and c = pivot lower in a plane of its own after the
// layout ([k * 4 groups + ch]); rows 6 and 7 hold in words 10 to 14 the SA row's coupling to
// the mean flow below and above.
constexpr int LW_WORDS = 15, LW_ROWS = 8, LW_CHAINS = 4;
__host__ __device__ __forceinline__ int line_groups(const Plan3Dev& p) { return (p.n_chains + LW_CHAINS - 1) / LW_CHAINS; }
__host__ __device__ __forceinline__ size_t line_words(const Plan3Dev& p) {
  return (size_t)p.chain_L * line_groups(p) * LW_WORDS * LW_ROWS * LW_CHAINS;
}

// The elimination down chain ch: T = D - lower C_{k-1}, P = T^-1 (Gauss-Jordan, one reciprocal a
// pivot), C = P upper, and the SA row's scalars, from the faces' terms (lam, mflux, dflux) and the
// cells' diagonals (dflow, dsa); its rows leave eight at a time.
template <class TF, bool SA>
__host__ __device__ __forceinline__ void line_factor_chain(const Plan3Dev& p, const double* __restrict__ U,
                                                           const double* __restrict__ lam,
                                                           const double* __restrict__ mflux,
                                                           const double* __restrict__ dflux,
                                                           const double* __restrict__ dflow,
                                                           const double* __restrict__ dsa, TF* __restrict__ F, int ch) {
  const double g = p.P.gamma;
  const int groups = line_groups(p), len = p.ch_len[ch];
  TF* out = F + ((size_t)(ch / LW_CHAINS) * LW_WORDS) * 32 + (ch % LW_CHAINS) * LW_ROWS;
  const size_t stride = (size_t)groups * LW_WORDS * 32;
  const bool coupled = SA && p.line_coupled;
  double C[5][5] = {}, q[NV3_MAX] = {}, qb[NV3_MAX] = {};   // this cell's state, the one below's
  double sl[3] = {0.0, 0.0, 0.0}, ll = 0.0, csa = 0.0, lsa = 0.0;   // the link below, outward from this cell
  bool linked = false;
  if (len > 0) prim_at_n<SA ? 6 : 5>(p, U, p.ch_cells[(size_t)ch * p.chain_L], q);
  for (int k = 0; k < len; ++k, out += stride) {
    const int c = p.ch_cells[(size_t)ch * p.chain_L + k];
    double T[5][5], L[5][5];
    if (linked) coupling5_closed(qb, sl[0], sl[1], sl[2], ll, g, L);
    else
#pragma unroll
      for (int a = 0; a < 5; ++a)
#pragma unroll
        for (int b = 0; b < 5; ++b) L[a][b] = 0.0;
    const double dg = dflow[c];
#pragma unroll
    for (int a = 0; a < 5; ++a)
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        double m = L[a][0] * C[0][b];
#pragma unroll
        for (int t = 1; t < 5; ++t) m = m + L[a][t] * C[t][b];
        T[a][b] = (a == b ? dg : 0.0) - m;
      }
    // the SA row's scalars beside the mean flow's blocks, and the coupled form's rows
    double slo = 0.0, spiv = 0.0, sc = 0.0, cpl[2][5] = {};
    if constexpr (SA) {
      if (!coupled) {
        slo = lsa;
        spiv = 1.0 / (dsa[c] - lsa * csa);
      } else if (linked) {
        sa_coupling_row(qb, sl, 1.0, cpl[0]);
      }
    }
    // word w of the rows: the first six, or all eight
    auto put = [&](int w, double r0, double r1, double r2, double r3, double r4, double r5, double r6, double r7) {
      TF* o = out + w * 32;
      if constexpr (sizeof(TF) == 4) {
        *reinterpret_cast<float4*>(o) = make_float4((float)r0, (float)r1, (float)r2, (float)r3);
        *reinterpret_cast<float4*>(o + 4) = make_float4((float)r4, (float)r5, (float)r6, (float)r7);
      } else {
        *reinterpret_cast<double2*>(o) = make_double2(r0, r1);
        *reinterpret_cast<double2*>(o + 2) = make_double2(r2, r3);
        *reinterpret_cast<double2*>(o + 4) = make_double2(r4, r5);
        if (coupled) *reinterpret_cast<double2*>(o + 6) = make_double2(r6, r7);
      }
    };
    // the link above: this cell's upper block and, for the next element, its lower one
    const int sign = k + 1 < len ? p.ch_sign[(size_t)ch * p.chain_L + k] : 0;
    double su[3] = {0.0, 0.0, 0.0}, lu = 0.0, qn[NV3_MAX] = {}, upsa = 0.0, nextsa = 0.0;
    if (k + 1 < len) prim_at_n<SA ? 6 : 5>(p, U, p.ch_cells[(size_t)ch * p.chain_L + k + 1], qn);
    if (sign != 0) {
      const int f = p.ch_face[(size_t)ch * p.chain_L + k];
      int fa, fi, fj, fk;
      face_of(p, f, fa, fi, fj, fk);
      face_vector(p, fa, fi, fj, fk, su);
#pragma unroll
      for (int m = 0; m < 3; ++m) su[m] *= (double)sign;
      lu = lam[f];
      if constexpr (SA) {
        const double um = -(double)sign * mflux[f], d = dflux[f];
        upsa = -((um > 0.0 ? um : 0.0) + d) / qn[0];
        nextsa = -((-um > 0.0 ? -um : 0.0) + d) / q[0];
        if (coupled) sa_coupling_row(qn, su, 1.0, cpl[1]);
      }
    }
    if constexpr (SA) {
      if (!coupled) csa = sc = spiv * upsa;
      lsa = nextsa;
    }
#pragma unroll
    for (int b = 0; b < 5; ++b) put(b, L[0][b], L[1][b], L[2][b], L[3][b], L[4][b], b == 0 ? slo : (b == 1 ? spiv : 0.0), 0.0, 0.0);
    // P = T^-1 in place
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const double inv = 1.0 / T[i][i];
      T[i][i] = 1.0;
#pragma unroll
      for (int b = 0; b < 5; ++b) T[i][b] = T[i][b] * inv;
#pragma unroll
      for (int a = 0; a < 5; ++a) {
        if (a == i) continue;
        const double f = T[a][i];
        T[a][i] = 0.0;
#pragma unroll
        for (int b = 0; b < 5; ++b) T[a][b] = T[a][b] - f * T[i][b];
      }
    }
#pragma unroll
    for (int b = 0; b < 5; ++b) put(5 + b, T[0][b], T[1][b], T[2][b], T[3][b], T[4][b], 0.0, 0.0, 0.0);
    // C = P upper
    if (sign != 0) {
      double B[5][5];
      coupling5_closed(qn, su[0], su[1], su[2], lu, g, B);
#pragma unroll
      for (int a = 0; a < 5; ++a)
#pragma unroll
        for (int b = 0; b < 5; ++b) {
          double m = T[a][0] * B[0][b];
#pragma unroll
          for (int t = 1; t < 5; ++t) m = m + T[a][t] * B[t][b];
          C[a][b] = m;
        }
    } else {
#pragma unroll
      for (int a = 0; a < 5; ++a)
#pragma unroll
        for (int b = 0; b < 5; ++b) C[a][b] = 0.0;
    }
#pragma unroll
    for (int b = 0; b < 5; ++b) put(10 + b, C[0][b], C[1][b], C[2][b], C[3][b], C[4][b], b == 0 ? sc : 0.0, cpl[0][b], cpl[1][b]);
    linked = sign != 0;
    ll = lu;
#pragma unroll
    for (int m = 0; m < 3; ++m) sl[m] = -su[m];
#pragma unroll
    for (int v = 0; v < NV3_MAX; ++v) {
      qb[v] = q[v];
      q[v] = qn[v];
    }
  }
  if constexpr (SA) {
    if (!coupled) return;
    // the SA chain from its far end: 1 / (d_k - upper_k c_{k+1}), c_k = that times lower_k
    TF* plane = F + line_words(p);
    double cs = 0.0;
    for (int k = len - 1; k >= 0; --k) {
      out -= stride;
      const size_t at = (size_t)ch * p.chain_L + k;
      const int c = p.ch_cells[at], up = k + 1 < len ? p.ch_sign[at] : 0, down = k > 0 ? p.ch_sign[at - 1] : 0;
      double u = 0.0, l = 0.0;
      if (up != 0) {
        const int f = p.ch_face[at];
        const double m = -(double)up * mflux[f];
        u = -((m > 0.0 ? m : 0.0) + dflux[f]) / U[p.ch_cells[at + 1]];
      }
      if (down != 0) {
        const int f = p.ch_face[at - 1];
        const double m = (double)down * mflux[f];
        l = -((m > 0.0 ? m : 0.0) + dflux[f]) / U[p.ch_cells[at - 1]];
      }
      const double piv = 1.0 / (dsa[c] - u * cs);
      cs = piv * l;
      out[10 * 32 + 5] = (TF)u;
      out[11 * 32 + 5] = (TF)piv;
      plane[(size_t)k * groups * LW_CHAINS + ch] = (TF)cs;
    }
  }
}

}  // namespace jr

namespace jr {

// The loads on wall face w (src/jaxrans/post/forces.py:48-68): 7 values -- the gauge
// pressure, the area vector into the fluid (3), the laminar viscous force on the body
// (3) -- from the ghost-filled primitive canvas Q.
inline __host__ __device__ void wall_load(const Plan3Dev& p, const double* Q, int w, double out[7]) {
  const int n = p.NI * p.NJ * p.NK;
  const double g = p.P.gamma;
  const int c = p.w_cell[w], a = p.w_family[w], f = p.w_face[w];
  const int fj = p.NJ + (a == 1), fk = p.NK + (a == 2);
  const int i = f / (fj * fk), j = (f / fk) % fj, k = f % fk;
  double s[3];
  face_vector(p, a, i, j, k, s);
  const double into = p.w_into[w];
  out[0] = Q[(size_t)4 * n + c] - 1.0 / g;
  for (int m = 0; m < 3; ++m) out[1 + m] = into * s[m];
  for (int m = 0; m < 3; ++m) out[4 + m] = 0.0;
  if (p.P.mu_inf > 0.0) {
    double grad[3][5];
    face_gradient<double, 4>(p, Q, a, i, j, k, grad);
    int lo[3] = {i, j, k};
    lo[a] -= 1;
    double ql[NV3_MAX], qh[NV3_MAX];
    load_cell(p, Q, cell_index(p, lo[0], lo[1], lo[2]), ql);
    load_cell(p, Q, cell_index(p, i, j, k), qh);
    const double T = 0.5 * (g * ql[4] / ql[0] + g * qh[4] / qh[0]);
    const double mu = viscosity3(p.P, T);
    const double div = grad[0][0] + grad[1][1] + grad[2][2];
    const double ttd = (2.0 / 3.0) * div;
    for (int comp = 0; comp < 3; ++comp) {
      double tau[3];
      for (int d = 0; d < 3; ++d) {
        if (comp == d) {
          tau[d] = mu * (2.0 * grad[comp][comp] - ttd);
        } else {
          const int lo2 = comp < d ? comp : d, hi2 = comp < d ? d : comp;
          tau[d] = mu * (grad[hi2][lo2] + grad[lo2][hi2]);
        }
      }
      out[4 + comp] = into * ((tau[0] * s[0] + tau[1] * s[1]) + tau[2] * s[2]);
    }
  }
}

}  // namespace jr
