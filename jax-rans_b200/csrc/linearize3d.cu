// The linearised 3D J.v on the device: the factors once per Newton step (k3_lin_faces,
// k3_lin_cells), and per Krylov vector the tangents of the primitive canvas (k3_tangents,
// ghosts included) and one tile kernel (k3_jv) that maps them to V/dt z + dR1/dU z.
#include "linearize3d.cuh"

namespace jr {

// One thread per face slot of the factors' layout (k fastest).  Bound by FP64 issue (the
// flux's ten columns, two an evaluation, which 255 registers hold without spills): 6.1 ms on
// the 3.9M-cell wing, once per Newton step.  A single product (jr_jvp3d) is therefore left to
// the dual-number J.v: factors and product together cost as much (8.5 against 8.0 ms there).
template <bool VISC, bool SA>
__global__ void __launch_bounds__(128) k3_lin_faces(Plan3Dev p, const double* __restrict__ Q,
                                                    double* __restrict__ lin) {
  const int row = lin_chunks(p) * LIN_K, nc = lin_factors(p);
  const size_t total = (size_t)3 * (p.NI + 1) * (p.NJ + 1) * row;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    const int k = (int)(e % row);
    const int r = (int)(e / row);
    const int j = r % (p.NJ + 1), i = (r / (p.NJ + 1)) % (p.NI + 1), a = r / ((p.NJ + 1) * (p.NI + 1));
    if (i >= p.NI + (a == 0) || j >= p.NJ + (a == 1) || k >= p.NK + (a == 2) || !face_live(p, a, i, j, k)) continue;
    linearize_face3<VISC, SA>(p, Q, a, i, j, k, lin + lin_at(p, nc, a, i, j, k));
  }
}

__global__ void __launch_bounds__(128) k3_lin_cells(Plan3Dev p, const double* __restrict__ Q, double* __restrict__ out) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    if (p.interior[c]) linearize_cell3(p, Q, c, out);
}

// The tangents of (rho, u, v, w, p[, nu~]) and T = gamma p / rho of every canvas cell
// along the conservative direction z, at the ghost-filled canvas Q of U: NV + 1 planes.
// Bound by its bytes (2 NV values read, NV + 1 written a cell), so eight blocks an SM: the
// few ghosts' conditions, not the cells, pay for the registers that costs (some spilled);
// 206 us on the 3.9M-cell wing against 344 us at 106 registers.
template <int NV>
__global__ void __launch_bounds__(128, 8) k3_tangents(Plan3Dev p, const double* __restrict__ U,
                                                   const double* __restrict__ Q, const double* __restrict__ z,
                                                   double* __restrict__ dq) {
  const int n = p.NI * p.NJ * p.NK;
  const double g = p.P.gamma;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    double t[NV3_MAX], inv, pr;
    const int gid = p.ghost_of[c];
    if (gid >= 0) {
      Dual q[NV3_MAX];
      ghost_state<NV>(p, U, z, gid, q);
#pragma unroll
      for (int v = 0; v < NV; ++v) t[v] = q[v].d;
      inv = 1.0 / q[0].v;
      pr = q[4].v;
    } else {
      double q[NV3_MAX], d[NV3_MAX];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        q[v] = Q[(size_t)v * n + c];
        d[v] = z[(size_t)v * n + c];
      }
      inv = 1.0 / q[0];
      t[0] = d[0];
#pragma unroll
      for (int m = 1; m < 4; ++m) t[m] = (d[m] - q[m] * d[0]) * inv;
      const double vv = (q[1] * q[1] + q[2] * q[2]) + q[3] * q[3];
      t[4] = (g - 1.0) * ((d[4] - ((q[1] * d[1] + q[2] * d[2]) + q[3] * d[3])) + 0.5 * vv * d[0]);
      if constexpr (NV > 5) t[5] = (d[5] - q[5] * d[0]) * inv;
      pr = q[4];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) dq[(size_t)v * n + c] = t[v];
    dq[(size_t)NV * n + c] = g * (t[4] - pr * inv * t[0]) * inv;
  }
}

// The tile of k3_jv: 4 x 8 x 8 cells.  The tangents of the tile and a ring of one cell, the
// tangents' node means and every face's flux stay in shared memory (93 KB, two CTAs an SM).
// Its 896 faces (5 x 8 x 8, 4 x 9 x 8, 4 x 8 x 9) are 28 warps' worth, four for each of the
// CTA's seven warps with no barrier between them.
constexpr int JT_I = 4, JT_J = 8, JT_K = 8, JT_THREADS = 224, JT_CELLS = JT_I * JT_J * JT_K;
constexpr int JH_J = JT_J + 2, JH_K = JT_K + 2, JH = (JT_I + 2) * JH_J * JH_K;
constexpr int JN_J = JT_J + 1, JN_K = JT_K + 1, JN = (JT_I + 1) * JN_J * JN_K;
constexpr int JF_I = (JT_I + 1) * JT_J * JT_K, JF_J = JT_I * (JT_J + 1) * JT_K, JF = JF_I + JF_J + JT_I * JT_J * (JT_K + 1);
static_assert(JT_K == LIN_K, "a tile's rows are the factors' chunks");

template <bool VISC, bool SA> struct JvTile {
  static constexpr int NV = SA ? 6 : 5;
  double dq[NV + 1][JH];
  double node[VISC ? (SA ? 5 : 4) : 1][VISC ? JN : 1];   // u, v, w, T[, nu~]
  double F[NV][JF];
  unsigned char in[JH];
};

// face e of a tile: its family and place
__device__ __forceinline__ void tile_face(int e, int& a, int& fi, int& fj, int& fk) {
  a = e < JF_I ? 0 : (e < JF_I + JF_J ? 1 : 2);
  e -= a == 0 ? 0 : (a == 1 ? JF_I : JF_I + JF_J);
  const int nk = JT_K + (a == 2), nj = JT_J + (a == 1);
  fk = e % nk;
  fj = (e / nk) % nj;
  fi = e / (nk * nj);
}

// the tangent flux of face (fi, fj, fk) of family a, in tile coordinates; hi, lo: its cells,
// x: its factors
template <bool VISC, bool SA>
__device__ __forceinline__ void jv_face3(const JvTile<VISC, SA>& t, const double* __restrict__ x, double gamma,
                                         bool qcr, int a, int fi, int fj, int fk, int hi, int lo, double* dF) {
  using X = Lin3<VISC, SA>;
  constexpr int NV = SA ? 6 : 5;
  auto f = [&](int c) { return __ldg(x + c * LIN_K); };
  double al[5], ah[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    al[v] = t.dq[v][lo];
    ah[v] = t.dq[v][hi];
  }
#pragma unroll
  for (int r = 0; r < 5; ++r) {
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < 5; ++s) acc += f(X::A + r * 10 + s) * al[s];
#pragma unroll
    for (int s = 0; s < 5; ++s) acc += f(X::A + r * 10 + 5 + s) * ah[s];
    dF[r] = acc;
  }
  if constexpr (SA) {
    const double mass = f(X::MASS);
    dF[NV - 1] = f(X::UP) * dF[0] + mass * (mass > 0.0 ? t.dq[5][lo] : t.dq[5][hi]);
  }
  if constexpr (VISC) {
    constexpr int NPHI = SA ? 5 : 4;
    const int n00 = (fi * JN_J + fj) * JN_K + fk;
    const int s1 = a == 0 ? JN_K : JN_J * JN_K, s2 = a == 2 ? JN_K : 1;   // along the face's two other axes
    double gr[3][NPHI], S[3];
    {
      double c23[3], c31[3], c12[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        c23[d] = f(X::GEO + d);
        c31[d] = f(X::GEO + 3 + d);
        c12[d] = f(X::GEO + 6 + d);
        S[d] = f(X::S + d);
      }
#pragma unroll
      for (int m = 0; m < NPHI; ++m) {
        constexpr int rows[5] = {1, 2, 3, NV, NV - 1};
        const double p1 = t.dq[rows[m]][hi] - t.dq[rows[m]][lo];
        const double p2 = t.node[m][n00 + s1 + s2] - t.node[m][n00];
        const double p3 = t.node[m][n00 + s2] - t.node[m][n00 + s1];
#pragma unroll
        for (int d = 0; d < 3; ++d) gr[d][m] = p1 * c23[d] + p2 * c31[d] + p3 * c12[d];
      }
    }
    const double dmul = f(X::DMU) * (0.5 * (t.dq[NV][lo] + t.dq[NV][hi]));
    double dmu = dmul, dk = dmul * (1.0 / (PR_LAMINAR * (gamma - 1.0)));
    double dmut = 0.0;
    if constexpr (SA) {
      const double dr = 0.5 * (al[0] + ah[0]), dp = 0.5 * (al[4] + ah[4]), dn = 0.5 * (t.dq[5][lo] + t.dq[5][hi]);
      dmut = (f(X::MUT) * dr + f(X::MUT + 1) * dp) + f(X::MUT + 2) * dn;
      dmu += dmut;
      dk += dmut * (1.0 / (PR_TURBULENT * (gamma - 1.0)));
      const double dcoef = (f(X::DCOEF) * dr + f(X::DCOEF + 1) * dp) + f(X::DCOEF + 2) * dn;
      const double dgn = (gr[0][NPHI - 1] * S[0] + gr[1][NPHI - 1] * S[1]) + gr[2][NPHI - 1] * S[2];
      dF[NV - 1] -= f(X::COEF) * dgn + dcoef * f(X::GN);
    }
    const double mu = f(X::MU), ttd = (2.0 / 3.0) * ((gr[0][0] + gr[1][1]) + gr[2][2]);
    double energy = dk * f(X::GT) + f(X::K) * ((gr[0][3] * S[0] + gr[1][3] * S[1]) + gr[2][3] * S[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double l = f(X::L + c);
      double dl = -ttd * S[c];
#pragma unroll
      for (int d = 0; d < 3; ++d) dl += (gr[d][c] + gr[c][d]) * S[d];
      double force = mu * l, dforce = mu * dl + l * dmu;
      if constexpr (SA) {
        if (qcr) {
          force += f(X::XF + c);
          dforce += f(X::XMU + c) * dmut;
#pragma unroll
          for (int e = 0; e < 9; ++e) dforce += f(X::XG + 9 * c + e) * gr[e / 3][e % 3];
        }
      }
      dF[1 + c] -= dforce;
      energy += 0.5 * (al[1 + c] + ah[1 + c]) * force + f(X::VEL + c) * dforce;
    }
    dF[4] -= energy;
  }
}

// w = vdt z + dR1/dU z on one tile of the canvas (rows outside the blocks: (vdt + 1) z).
// A Krylov vector of the 3.9M-cell wing (SA, 13.5M faces) reads 656 bytes of factors a face:
// 2.19 ms a product, 4.1 TB/s of factors (the dual-number J.v it replaces in the Newton step,
// bound by FP64 divisions and roots: 8.0 ms; family by family with barriers between, 320
// threads and spills: 2.63 ms; that with the next family prefetched into L2: 3.03 ms).
// On a 49k-cell wing, 390 tiles, it is latency: 61 us.
template <bool VISC, bool SA>
__global__ void __launch_bounds__(JT_THREADS, 2)
    k3_jv(Plan3Dev p, const double* __restrict__ lin, const double* __restrict__ lcell, const double* __restrict__ dq,
          const double* __restrict__ z, const double* __restrict__ vdt, double* __restrict__ w) {
  using Tile = JvTile<VISC, SA>;
  using X = Lin3<VISC, SA>;
  constexpr int NV = Tile::NV;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Tile& t = *reinterpret_cast<Tile*>(smem_raw);
  const int n = p.NI * p.NJ * p.NK, nc = lin_factors(p);
  const int k0 = blockIdx.x * JT_K, i0 = blockIdx.y * JT_I, j0 = blockIdx.z * JT_J;
  const int tid = threadIdx.x;
  // 1. the tangents of the tile and its ring (indices clamped to the canvas)
  int any = 0;
  for (int e = tid; e < JH; e += JT_THREADS) {
    const int i = i0 - 1 + e / (JH_J * JH_K), j = j0 - 1 + (e / JH_K) % JH_J, k = k0 - 1 + e % JH_K;
    const int c = cell_index(p, i, j, k);
    const bool in = i >= 0 && i < p.NI && j >= 0 && j < p.NJ && k >= 0 && k < p.NK && p.interior[c];
    t.in[e] = in;
    any |= in;
#pragma unroll
    for (int v = 0; v <= NV; ++v)
      if (VISC || v < NV) t.dq[v][e] = dq[(size_t)v * n + c];
  }
  any = __syncthreads_or(any);
  if (any) {
    // 2. the nodes' means of their eight cells
    if constexpr (VISC) {
      constexpr int NPHI = SA ? 5 : 4;
      for (int e = tid; e < JN; e += JT_THREADS) {
        // cell (-1, -1, -1) of the eight
        const int h = ((e / (JN_J * JN_K)) * JH_J + (e / JN_K) % JN_J) * JH_K + e % JN_K;
#pragma unroll
        for (int m = 0; m < NPHI; ++m) {
          constexpr int rows[5] = {1, 2, 3, NV, NV - 1};
          const double* q = t.dq[rows[m]] + h;
          double s[2];
#pragma unroll
          for (int d = 0; d < 2; ++d)
            s[d] = (q[d] + q[JH_J * JH_K + d]) + (q[JH_K + d] + q[JH_J * JH_K + JH_K + d]);
          t.node[m][e] = 0.125 * (s[0] + s[1]);
        }
      }
      __syncthreads();
    }
    // 3. the faces' tangent fluxes
    const bool qcr = SA && p.P.c_cr1 != 0.0;
#pragma unroll 1
    for (int e = tid; e < JF; e += JT_THREADS) {
      int a, fi, fj, fk;
      tile_face(e, a, fi, fj, fk);
      const int hi = ((fi + 1) * JH_J + fj + 1) * JH_K + fk + 1;
      const int lo = hi - (a == 0 ? JH_J * JH_K : (a == 1 ? JH_K : 1));
      if (!t.in[hi] && !t.in[lo]) continue;
      double dF[NV];
      jv_face3<VISC, SA>(t, lin + lin_at(p, nc, a, i0 + fi, j0 + fj, k0 + fk), p.P.gamma, qcr, a, fi, fj, fk, hi, lo, dF);
#pragma unroll
      for (int v = 0; v < NV; ++v) t.F[v][e] = dF[v];
    }
    __syncthreads();
  }
  // 4. the cells' sums
  for (int e = tid; e < JT_CELLS; e += JT_THREADS) {
    const int ci = e / (JT_J * JT_K), cj = (e / JT_K) % JT_J, ck = e % JT_K;
    const int i = i0 + ci, j = j0 + cj, k = k0 + ck;
    if (i >= p.NI || j >= p.NJ || k >= p.NK) continue;
    const int h = ((ci + 1) * JH_J + cj + 1) * JH_K + ck + 1;
    const int c = (i * p.NJ + j) * p.NK + k;
    const bool mine = t.in[h];
    double acc[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    if (mine) {
      double curl[3] = {0.0, 0.0, 0.0}, gn[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int nk = JT_K + (a == 2), nj = JT_J + (a == 1);
        const int lo = (a == 0 ? 0 : (a == 1 ? JF_I : JF_I + JF_J)) + (ci * nj + cj) * nk + ck;
        const int hi = lo + (a == 0 ? nj * nk : (a == 1 ? nk : 1));
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] += t.F[v][hi] - t.F[v][lo];
        if constexpr (SA) {
          const int step = a == 0 ? JH_J * JH_K : (a == 1 ? JH_K : 1);
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            const int o = side ? h + step : h - step;
            const double half = side ? 0.5 : -0.5;
            const double* s = lin + lin_at(p, nc, a, i + (a == 0) * side, j + (a == 1) * side, k + (a == 2) * side) +
                              X::S * LIN_K;
            double v[3], S[3];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
              v[m] = half * (t.dq[1 + m][h] + t.dq[1 + m][o]);
              S[m] = __ldg(s + m * LIN_K);
            }
            const double nu = half * (t.dq[5][h] + t.dq[5][o]);
            curl[0] += S[1] * v[2] - S[2] * v[1];
            curl[1] += S[2] * v[0] - S[0] * v[2];
            curl[2] += S[0] * v[1] - S[1] * v[0];
#pragma unroll
            for (int m = 0; m < 3; ++m) gn[m] += nu * S[m];
          }
        }
      }
      if constexpr (SA) {
        double src = (lcell[c] * t.dq[0][h] + lcell[(size_t)n + c] * t.dq[4][h]) + lcell[(size_t)2 * n + c] * t.dq[5][h];
#pragma unroll
        for (int m = 0; m < 3; ++m)
          src += lcell[(size_t)(3 + m) * n + c] * curl[m] + lcell[(size_t)(6 + m) * n + c] * gn[m];
        acc[NV - 1] -= src;
      }
    }
    const double a = vdt[c];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const double zc = z[(size_t)v * n + c];
      w[(size_t)v * n + c] = a * zc + (mine ? acc[v] : zc);
    }
  }
}

// ---- launchers
// the doubles of the factors' buffers: faces, cells, and the tangents of one vector
void lin3_sizes(const Plan3Dev& p, size_t& face, size_t& cell, size_t& tangents) {
  const size_t n = (size_t)p.NI * p.NJ * p.NK;
  face = lin_words(p);
  cell = p.nvar > 5 ? LIN_CELL * n : 0;
  tangents = (size_t)(p.nvar + 1) * n;
}

template <bool VISC, bool SA> static void lin_faces(const Plan3Dev& p, const double* Q, double* face, cudaStream_t st) {
  const size_t total = (size_t)3 * (p.NI + 1) * (p.NJ + 1) * lin_chunks(p) * LIN_K;
  k3_lin_faces<VISC, SA><<<(unsigned)((total + 127) / 128), 128, 0, st>>>(p, Q, face);
}

// The factors at U into face and cell; Q (nvar canvas planes) is left as U's ghost-filled
// primitive canvas, which launch_lin_jv3 reads.
void launch_linearize3(const Plan3Dev& p, const double* U, double* Q, double* face, double* cell, cudaStream_t st) {
  launch_canvas3(p, U, Q, st);
  if (p.P.mu_inf > 0.0) launch_nodes3(p, Q, st);
  counted3(p.nvar > 5 ? 2 : 1);
  if (p.nvar > 5) {
    lin_faces<true, true>(p, Q, face, st);
    k3_lin_cells<<<(p.NI * p.NJ * p.NK + 127) / 128, 128, 0, st>>>(p, Q, cell);
  } else if (p.P.mu_inf > 0.0) {
    lin_faces<true, false>(p, Q, face, st);
  } else {
    lin_faces<false, false>(p, Q, face, st);
  }
}

template <bool VISC, bool SA>
static void jv_tile(const Plan3Dev& p, const double* face, const double* cell, const double* dq, const double* z,
                    const double* vdt, double* w, cudaStream_t st) {
  const dim3 grid((p.NK + JT_K - 1) / JT_K, (p.NI + JT_I - 1) / JT_I, (p.NJ + JT_J - 1) / JT_J);
  const int bytes = (int)sizeof(JvTile<VISC, SA>);
  cudaFuncSetAttribute(k3_jv<VISC, SA>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  k3_jv<VISC, SA><<<grid, JT_THREADS, bytes, st>>>(p, face, cell, dq, z, vdt, w);
}

// w = vdt z + dR1/dU z from the factors launch_linearize3 stored
void launch_lin_jv3(const Plan3Dev& p, const double* U, const double* Q, const double* face, const double* cell,
                    double* dq, const double* z, const double* vdt, double* w, cudaStream_t st) {
  const int blocks = (p.NI * p.NJ * p.NK + 127) / 128;
  counted3(2);
  if (p.nvar > 5) {
    k3_tangents<6><<<blocks, 128, 0, st>>>(p, U, Q, z, dq);
    jv_tile<true, true>(p, face, cell, dq, z, vdt, w, st);
  } else {
    k3_tangents<5><<<blocks, 128, 0, st>>>(p, U, Q, z, dq);
    if (p.P.mu_inf > 0.0) jv_tile<true, false>(p, face, cell, dq, z, vdt, w, st);
    else jv_tile<false, false>(p, face, cell, dq, z, vdt, w, st);
  }
}

}  // namespace jr
