// Test only: the 3D kernels' host-and-device bodies (jax-rans_b200/csrc/residual3d.cuh,
// linesolve3d.cuh, linearize3d.cuh) run on the host on a plan given by its C-ABI descriptor -- the
// same bodies in the kernels' order, loops in place of threads -- a check of the kernels' indexing
// and arithmetic without a GPU.  What has no such body (the line solve's sweeps and the tile that
// applies the stored factors, which work across a warp or a block) is restated here over the
// device's layout.  Nothing of the library calls this; it is built by tests/conftest.py.
#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "../../jax-rans_b200/csrc/plan3d_desc.cuh"
#include "../../jax-rans_b200/csrc/linearize3d.cuh"
#include "../../jax-rans_b200/csrc/linesolve3d.cuh"
#include "../../jax-rans_b200/csrc/newton3d.cuh"
#include "../../jax-rans_b200/csrc/walldist3d.cuh"

using namespace jr;

// A plan over the descriptor's arrays and the tables made from it
struct HostPlan {
  Plan3Dev p{};
  std::vector<int> ghost_of, root, off, rec, len, offchain;
  std::vector<double> geo;
  std::vector<Dual> nodes;
};

static void plan_of(const jr_plan3d_desc* d, HostPlan& h) {
  Plan3Dev& p = h.p;
  p.NI = d->NI;
  p.NJ = d->NJ;
  p.NK = d->NK;
  p.nvar = d->nvar;
  p.interior = d->interior;
  p.volume = d->volume;
  for (int a = 0; a < 3; ++a) p.faces[a] = d->faces[a];
  p.centres = d->centres;
  p.distance = d->distance;
  p.g_kind = d->kind;
  p.g_normal = d->normal;
  p.neighbours = d->neighbours;
  p.n_chains = d->n_chains;
  p.line_fp32 = d->line_precision;
  p.line_coupled = d->preconditioner == 2;
  p.chain_L = d->chain_L;
  p.ch_cells = d->chain_cells;
  p.ch_face = d->chain_up_face;
  p.ch_sign = d->chain_up_sign;
  p.n_walls = d->n_walls;
  p.w_cell = d->wall_cell;
  p.w_family = d->wall_family;
  p.w_face = d->wall_face;
  p.w_into = d->wall_into;
  physics3_from_desc(p.P, d);
  const size_t n = (size_t)d->NI * d->NJ * d->NK;
  ghost_programs(d, n, h.ghost_of, h.root, h.off, h.rec);
  p.ghost_of = h.ghost_of.data();
  p.gp_root = h.root.data();
  p.gp_off = h.off.data();
  p.gp_rec = h.rec.data();
  chain_tables(d, n, h.len, h.offchain);
  p.ch_len = h.len.data();
  p.n_offchain = (int)h.offchain.size();
  p.offchain = h.offchain.data();
  if (p.P.mu_inf > 0.0) {   // k3_face_geometry
    const size_t nf = (size_t)face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
    h.geo.resize(10 * nf);
    for (size_t f = 0; f < nf; ++f) {
      int a, i, j, k;
      double g[10];
      face_of(p, (int)f, a, i, j, k);
      face_gradient_geometry(p, a, i, j, k, g);
      for (int q = 0; q < 10; ++q) h.geo[q * nf + f] = g[q];
    }
    p.face_geo = h.geo.data();
    h.nodes.resize((size_t)5 * node_count(p));
    p.node_buf = h.nodes.data();
  }
}

// k3_canvas: the ghost-filled primitive canvas, each ghost by its program
template <class T, int NV>
static void canvas_n(const Plan3Dev& p, const double* U, const double* dU, T* Q) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = 0; c < n; ++c) {
    if (p.ghost_of[c] < 0) {
      prim_cell_n<NV>(p, U, dU, Q, c);
      continue;
    }
    T q[NV3_MAX];
    ghost_state<NV>(p, U, dU, p.ghost_of[c], q);
    for (int v = 0; v < NV; ++v) Q[(size_t)v * n + c] = q[v];
  }
}

template <class T> static std::vector<T> canvas(const Plan3Dev& p, const double* U, const double* dU) {
  std::vector<T> Q((size_t)p.nvar * p.NI * p.NJ * p.NK);
  if (p.nvar > 5) canvas_n<T, 6>(p, U, dU, Q.data());
  else canvas_n<T, 5>(p, U, dU, Q.data());
  return Q;
}

// k3_node_phi, into p.node_buf
template <class T> static void node_values(const Plan3Dev& p, const T* Q) {
  if (!(p.P.mu_inf > 0.0)) return;
  T* nb = static_cast<T*>(p.node_buf);
  const int nn = node_count(p);
  for (int e = 0; e < nn; ++e) {
    const int I = e / ((p.NJ + 1) * (p.NK + 1)), J = (e / (p.NK + 1)) % (p.NJ + 1), K = e % (p.NK + 1);
    for (int m = 0; m < (p.nvar > 5 ? 5 : 4); ++m) nb[(size_t)m * nn + e] = node_phi_m(p, Q, I, J, K, m);
  }
}

// The ghost stages as the descriptor defines them, each from a copy of the canvas: what the ghost
// programs must give
static void fill_staged(const Plan3Dev& p, const jr_plan3d_desc* d, std::vector<double>& A) {
  const int n = p.NI * p.NJ * p.NK;
  int at = 0;
  for (int s = 0; s < d->n_stages; ++s) {
    const std::vector<double> in = A;
    for (int r = at; r < at + d->stage_records[s]; ++r) {
      double q[NV3_MAX], o[NV3_MAX];
      for (int v = 0; v < p.nvar; ++v) q[v] = in[(size_t)v * n + d->source[r]];
      condition3(d->kind[r], q, d->normal[3 * r], d->normal[3 * r + 1], d->normal[3 * r + 2], p.P, p.nvar, o);
      for (int v = 0; v < p.nvar; ++v) A[(size_t)v * n + d->ghost[r]] = o[v];
    }
    at += d->stage_records[s];
  }
}

// The residual: the device's two phases (every face once into a buffer, unwritten entries NaN, a
// viscous dual-number flux in its two parts; then the cell sums), or fused, each cell from its six
// faces' whole fluxes
template <class T, bool VISC, bool SA>
static void run(const Plan3Dev& p, const double* U, const double* dU, double* R, int first_order, bool fused) {
  const int n = p.NI * p.NJ * p.NK, nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  const std::vector<T> Q = canvas<T>(p, U, dU);
  node_values(p, Q.data());
  std::vector<double> F((size_t)p.nvar * nf, std::nan(""));
  if (!fused) {
    for (int f = 0; f < nf; ++f) {
      if constexpr (VISC && sizeof(T) == sizeof(Dual)) {
        store_face_flux<T, VISC, SA, 0, 1>(p, Q.data(), first_order, f, F.data(), (size_t)nf);
        store_face_flux<T, VISC, SA, 0, 2>(p, Q.data(), first_order, f, F.data(), (size_t)nf);
      } else {
        store_face_flux<T, VISC, SA>(p, Q.data(), first_order, f, F.data(), (size_t)nf);
      }
    }
    for (int c = 0; c < n; ++c) residual_cell_from_faces<T, SA>(p, Q.data(), F.data(), (size_t)nf, U, dU, R, c);
    return;
  }
  for (int c = 0; c < n; ++c) {
    if (p.interior[c]) {
      const int i = c / (p.NJ * p.NK), j = (c / p.NK) % p.NJ, k = c % p.NK;
      for (int a = 0; a < 3; ++a)
        for (int side = 0; side < 2; ++side) {
          const int fi = i + (a == 0) * side, fj = j + (a == 1) * side, fk = k + (a == 2) * side;
          T flux[NV3_MAX];
          face_flux<T, VISC, SA>(p, Q.data(), a, fi, fj, fk, first_order != 0, flux);
          for (int v = 0; v < p.nvar; ++v)
            F[(size_t)v * nf + face_flat(p, a, fi, fj, fk)] = tangent_or_value(flux[v]);
        }
    }
    residual_cell_from_faces<T, SA>(p, Q.data(), F.data(), (size_t)nf, U, dU, R, c);
  }
}

static int eval(const Plan3Dev& p, const double* U, const double* dU, double* R, int first_order, bool fused) {
  const bool visc = p.P.mu_inf > 0.0, sa = p.nvar > 5;
  if (dU) {
    if (sa) run<Dual, true, true>(p, U, dU, R, 1, fused);
    else if (visc) run<Dual, true, false>(p, U, dU, R, 1, fused);
    else run<Dual, false, false>(p, U, dU, R, 1, fused);
  } else {
    if (sa) run<double, true, true>(p, U, nullptr, R, first_order, fused);
    else if (visc) run<double, true, false>(p, U, nullptr, R, first_order, fused);
    else run<double, false, false>(p, U, nullptr, R, first_order, fused);
  }
  return 0;
}

// the device's two-phase form of jr3_host_eval
extern "C" int jr3_host_eval_faces(const jr_plan3d_desc* d, const double* U, const double* dU, double* R,
                                   int first_order) {
  HostPlan h;
  plan_of(d, h);
  return eval(h.p, U, dU, R, first_order, false);
}

extern "C" int jr3_host_eval(const jr_plan3d_desc* d, const double* U, const double* dU, double* R,
                             int first_order) {
  HostPlan h;
  plan_of(d, h);
  return eval(h.p, U, dU, R, first_order, true);
}

extern "C" int jr3_host_wave_speeds(const jr_plan3d_desc* d, const double* U, double* lam) {
  HostPlan h;
  plan_of(d, h);
  const Plan3Dev& p = h.p;
  const int total = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  for (int f = 0; f < total; ++f) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    lam[f] = wave_speed(p, U, a, i, j, k);
  }
  return 0;
}

// ---- the line solve: the kernels' bodies for the faces, the cells and the elimination, then the
// sweeps over the factor in its layout (k3_line_apply)
struct LineTerms {
  std::vector<double> lam, m, d, dflow, dsa, sum;
};

template <bool SA> static void line_terms(const Plan3Dev& p, const double* U, double cfl, LineTerms& t) {
  const int n = p.NI * p.NJ * p.NK, nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  t.lam.assign(nf, 0.0);
  t.m.assign(nf, 0.0);
  t.d.assign(nf, 0.0);
  t.dflow.assign(n, 0.0);
  t.dsa.assign(n, 0.0);
  t.sum.assign(n, 0.0);
  for (int f = 0; f < nf; ++f) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    line_face_terms<SA>(p, U, a, i, j, k, t.lam[f], t.m[f], t.d[f]);
  }
  for (int c = 0; c < n; ++c) {
    line_cell_terms<SA>(p, U, t.lam.data(), t.m.data(), t.d.data(), cfl, c, t.sum[c], t.dsa[c]);
    t.dflow[c] = t.sum[c] * (1.0 / cfl + 0.5);
  }
}

template <class TF, bool SA>
static void line_solve(const Plan3Dev& p, const double* U, double cfl, const double* r, double* z) {
  const size_t n = (size_t)p.NI * p.NJ * p.NK;
  const int groups = line_groups(p);
  const bool coupled = SA && p.line_coupled;
  LineTerms t;
  line_terms<SA>(p, U, cfl, t);
  std::vector<TF> F(line_words(p) + (size_t)p.chain_L * groups * LW_CHAINS);
  for (int ch = 0; ch < p.n_chains; ++ch)
    line_factor_chain<TF, SA>(p, U, t.lam.data(), t.m.data(), t.d.data(), t.dflow.data(), t.dsa.data(), F.data(), ch);
  for (int c = 0; c < p.n_offchain; ++c)
    for (int v = 0; v < p.nvar; ++v) z[v * n + p.offchain[c]] = r[v * n + p.offchain[c]];
  for (int ch = 0; ch < p.n_chains; ++ch) {
    const int len = p.ch_len[ch];
    const int* cells = p.ch_cells + (size_t)ch * p.chain_L;
    auto word = [&](int k, int w, int row) {
      return F[((((size_t)k * groups + ch / LW_CHAINS) * LW_WORDS + w) * LW_CHAINS + ch % LW_CHAINS) * LW_ROWS + row];
    };
    auto dot = [&](int k, int w, int row, const TF* x) {
      TF m = word(k, w, row) * x[0];
      for (int b = 1; b < 5; ++b) m = m + word(k, w + b, row) * x[b];
      return m;
    };
    std::vector<TF> x((size_t)(len + 1) * 6, TF(0));   // [element][row]; beyond the end: 0
    TF below[5] = {}, sbelow = TF(0);
    for (int k = 0; k < len; ++k) {
      TF rhs[5];
      for (int a = 0; a < 5; ++a) rhs[a] = TF(r[a * n + cells[k]]) - dot(k, 0, a, below);
      for (int a = 0; a < 5; ++a) x[k * 6 + a] = dot(k, 5, a, rhs);
      for (int a = 0; a < 5; ++a) below[a] = x[k * 6 + a];
      if (SA && !coupled) sbelow = x[k * 6 + 5] = word(k, 1, 5) * (TF(r[5 * n + cells[k]]) - word(k, 0, 5) * sbelow);
    }
    for (int k = len - 1; k >= 0; --k) {
      TF above[5];
      for (int a = 0; a < 5; ++a) above[a] = x[(k + 1) * 6 + a];
      for (int a = 0; a < 5; ++a) x[k * 6 + a] = x[k * 6 + a] - dot(k, 10, a, above);
      if (SA && !coupled) x[k * 6 + 5] = x[k * 6 + 5] - word(k, 10, 5) * x[(k + 1) * 6 + 5];
    }
    if (coupled) {
      for (int k = len - 1; k >= 0; --k) {
        const TF lo = k > 0 ? dot(k, 10, 6, &x[(k - 1) * 6]) : TF(0);
        const TF up = k + 1 < len ? dot(k, 10, 7, &x[(k + 1) * 6]) : TF(0);
        x[k * 6 + 5] = word(k, 11, 5) * ((TF(r[5 * n + cells[k]]) - (lo + up)) - word(k, 10, 5) * x[(k + 1) * 6 + 5]);
      }
      const TF* plane = F.data() + line_words(p) + ch;
      for (int k = 1; k < len; ++k) x[k * 6 + 5] = x[k * 6 + 5] - plane[(size_t)k * groups * LW_CHAINS] * x[(k - 1) * 6 + 5];
    }
    for (int k = 0; k < len; ++k)
      for (int v = 0; v < p.nvar; ++v) z[v * n + cells[k]] = double(x[k * 6 + v]);
  }
}

static void line_solve_as(const Plan3Dev& p, const double* U, double cfl, const double* r, double* z) {
  if (p.nvar > 5) {
    if (p.line_fp32) line_solve<float, true>(p, U, cfl, r, z);
    else line_solve<double, true>(p, U, cfl, r, z);
  } else {
    if (p.line_fp32) line_solve<float, false>(p, U, cfl, r, z);
    else line_solve<double, false>(p, U, cfl, r, z);
  }
}

extern "C" int jr3_host_precondition(const jr_plan3d_desc* d, const double* U, double cfl, const double* r,
                                     double* z) {
  HostPlan h;
  plan_of(d, h);
  line_solve_as(h.p, U, cfl, r, z);
  return 0;
}

// ---- the linearised J.v: the kernels' factors, applied as k3_tangents and k3_jv apply them
struct Linearised {
  std::vector<double> face, cell;
};

template <bool VISC, bool SA> static void linearise(const Plan3Dev& p, const double* U, Linearised& l) {
  const int n = p.NI * p.NJ * p.NK, nc = lin_factors(p);
  const std::vector<double> Q = canvas<double>(p, U, nullptr);
  node_values(p, Q.data());
  l.face.assign(lin_words(p), std::nan(""));
  l.cell.assign((size_t)LIN_CELL * n, std::nan(""));
  for (int a = 0; a < 3; ++a)
    for (int i = 0; i < p.NI + (a == 0); ++i)
      for (int j = 0; j < p.NJ + (a == 1); ++j)
        for (int k = 0; k < p.NK + (a == 2); ++k)
          if (face_live(p, a, i, j, k))
            linearize_face3<VISC, SA>(p, Q.data(), a, i, j, k, l.face.data() + lin_at(p, nc, a, i, j, k));
  if (SA)
    for (int c = 0; c < n; ++c)
      if (p.interior[c]) linearize_cell3(p, Q.data(), c, l.cell.data());
}

template <bool VISC, bool SA>
static void lin_jv(const Plan3Dev& p, const Linearised& l, const double* U, const double* z, double* w) {
  using X = Lin3<VISC, SA>;
  constexpr int NV = SA ? 6 : 5, NPHI = SA ? 5 : 4;
  const int n = p.NI * p.NJ * p.NK, nc = lin_factors(p);
  const double g = p.P.gamma;
  const std::vector<Dual> Q = canvas<Dual>(p, U, z);
  auto dq = [&](int v, int c) {   // the tangents of (rho, u, v, w, p[, nu~]) and, v == NV, of T
    return v < NV ? Q[(size_t)v * n + c].d : (g * Q[(size_t)4 * n + c] / Q[c]).d;
  };
  const int rows[5] = {1, 2, 3, NV, NV - 1};
  auto node = [&](int m, int I, int J, int K) {
    double s = 0.0;
    for (int e = 0; e < 8; ++e) s += dq(rows[m], cell_index(p, I - (e & 1), J - ((e >> 1) & 1), K - (e >> 2)));
    return 0.125 * s;
  };
  auto flux = [&](int a, int i, int j, int k, double* dF) {
    const double* x = l.face.data() + lin_at(p, nc, a, i, j, k);
    auto f = [&](int c) { return x[(size_t)c * LIN_K]; };
    const int lo = cell_index(p, i - (a == 0), j - (a == 1), k - (a == 2)), hi = cell_index(p, i, j, k);
    for (int r = 0; r < 5; ++r) {
      dF[r] = 0.0;
      for (int s = 0; s < 5; ++s) dF[r] += f(X::A + 10 * r + s) * dq(s, lo) + f(X::A + 10 * r + 5 + s) * dq(s, hi);
    }
    if (SA) dF[NV - 1] = f(X::UP) * dF[0] + f(X::MASS) * dq(5, f(X::MASS) > 0.0 ? lo : hi);
    if (!VISC) return;
    // the velocity, temperature (and nu~) gradients' tangents at the face
    const int n1[3] = {i + (a != 0), j + (a == 0), k}, n2[3] = {i, j + (a == 2), k + (a != 2)};
    double gr[3][5], S[3];
    for (int e = 0; e < 3; ++e) S[e] = f(X::S + e);
    for (int m = 0; m < NPHI; ++m) {
      const double p1 = dq(rows[m], hi) - dq(rows[m], lo);
      const double p2 = node(m, n1[0] + n2[0] - i, n1[1] + n2[1] - j, n1[2] + n2[2] - k) - node(m, i, j, k);
      const double p3 = node(m, n2[0], n2[1], n2[2]) - node(m, n1[0], n1[1], n1[2]);
      for (int e = 0; e < 3; ++e)
        gr[e][m] = p1 * f(X::GEO + e) + p2 * f(X::GEO + 3 + e) + p3 * f(X::GEO + 6 + e);
    }
    auto mean = [&](int v) { return 0.5 * (dq(v, lo) + dq(v, hi)); };
    const double dmul = f(X::DMU) * mean(NV);
    double dmu = dmul, dk = dmul / (PR_LAMINAR * (g - 1.0)), dmut = 0.0;
    if (SA) {
      dmut = f(X::MUT) * mean(0) + f(X::MUT + 1) * mean(4) + f(X::MUT + 2) * mean(5);
      dmu += dmut;
      dk += dmut / (PR_TURBULENT * (g - 1.0));
      const double dcoef = f(X::DCOEF) * mean(0) + f(X::DCOEF + 1) * mean(4) + f(X::DCOEF + 2) * mean(5);
      dF[NV - 1] -= f(X::COEF) * (gr[0][4] * S[0] + gr[1][4] * S[1] + gr[2][4] * S[2]) + dcoef * f(X::GN);
    }
    double energy = dk * f(X::GT) + f(X::K) * (gr[0][3] * S[0] + gr[1][3] * S[1] + gr[2][3] * S[2]);
    for (int c = 0; c < 3; ++c) {
      double dl = -(2.0 / 3.0) * (gr[0][0] + gr[1][1] + gr[2][2]) * S[c];
      for (int e = 0; e < 3; ++e) dl += (gr[e][c] + gr[c][e]) * S[e];
      double force = f(X::MU) * f(X::L + c), dforce = f(X::MU) * dl + f(X::L + c) * dmu;
      if (SA && p.P.c_cr1 != 0.0) {
        force += f(X::XF + c);
        dforce += f(X::XMU + c) * dmut;
        for (int e = 0; e < 9; ++e) dforce += f(X::XG + 9 * c + e) * gr[e / 3][e % 3];
      }
      dF[1 + c] -= dforce;
      energy += mean(1 + c) * force + f(X::VEL + c) * dforce;
    }
    dF[4] -= energy;
  };
  for (int c = 0; c < n; ++c) {
    if (!p.interior[c]) {
      for (int v = 0; v < NV; ++v) w[(size_t)v * n + c] = z[(size_t)v * n + c];
      continue;
    }
    const int i = c / (p.NJ * p.NK), j = (c / p.NK) % p.NJ, k = c % p.NK;
    double acc[NV] = {}, curl[3] = {}, gn[3] = {};
    for (int a = 0; a < 3; ++a)
      for (int side = 0; side < 2; ++side) {
        const int o = side ? 1 : -1, fi = i + (a == 0) * side, fj = j + (a == 1) * side, fk = k + (a == 2) * side;
        double dF[NV];
        flux(a, fi, fj, fk, dF);
        for (int v = 0; v < NV; ++v) acc[v] += o * dF[v];
        if (!SA) continue;
        const int nb = cell_index(p, i + (a == 0) * o, j + (a == 1) * o, k + (a == 2) * o);
        double S[3], v[3];
        face_vector(p, a, fi, fj, fk, S);
        for (int m = 0; m < 3; ++m) v[m] = 0.5 * o * (dq(1 + m, c) + dq(1 + m, nb));
        curl[0] += S[1] * v[2] - S[2] * v[1];
        curl[1] += S[2] * v[0] - S[0] * v[2];
        curl[2] += S[0] * v[1] - S[1] * v[0];
        for (int m = 0; m < 3; ++m) gn[m] += 0.5 * o * (dq(5, c) + dq(5, nb)) * S[m];
      }
    if (SA) {
      const double* s = l.cell.data() + c;
      double src = s[0] * dq(0, c) + s[n] * dq(4, c) + s[(size_t)2 * n] * dq(5, c);
      for (int m = 0; m < 3; ++m) src += s[(size_t)(3 + m) * n] * curl[m] + s[(size_t)(6 + m) * n] * gn[m];
      acc[NV - 1] -= src;
    }
    for (int v = 0; v < NV; ++v) w[(size_t)v * n + c] = acc[v];
  }
}

static void linearise_as(const Plan3Dev& p, const double* U, Linearised& l) {
  if (p.nvar > 5) linearise<true, true>(p, U, l);
  else if (p.P.mu_inf > 0.0) linearise<true, false>(p, U, l);
  else linearise<false, false>(p, U, l);
}

static void lin_jv_as(const Plan3Dev& p, const Linearised& l, const double* U, const double* z, double* w) {
  if (p.nvar > 5) lin_jv<true, true>(p, l, U, z, w);
  else if (p.P.mu_inf > 0.0) lin_jv<true, false>(p, l, U, z, w);
  else lin_jv<false, false>(p, l, U, z, w);
}

// J.v through the stored factors
extern "C" int jr3_host_lin_jvp(const jr_plan3d_desc* d, const double* U, const double* v, double* Jv) {
  HostPlan h;
  plan_of(d, h);
  Linearised l;
  linearise_as(h.p, U, l);
  lin_jv_as(h.p, l, U, v, Jv);
  return 0;
}

// The line solve's terms by face and cell, and the couplings along every link, against the forms
// they restate: the largest difference over the largest value of (lambda, the SA face terms left
// out where there are none, the flux Jacobian).  out: lambda, Jacobian.
extern "C" int jr3_host_line_terms(const jr_plan3d_desc* d, const double* U, double* out) {
  HostPlan h;
  plan_of(d, h);
  const Plan3Dev& p = h.p;
  const int nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  LineTerms t;
  if (p.nvar > 5) line_terms<true>(p, U, 25.0, t);
  else line_terms<false>(p, U, 25.0, t);
  double worst = 0.0, scale = 0.0, jworst = 0.0, jscale = 0.0;
  for (int f = 0; f < nf; ++f) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    const double lam = wave_speed(p, U, a, i, j, k);
    worst = std::fmax(worst, std::fabs(lam - t.lam[f]));
    scale = std::fmax(scale, lam);
    // A by forward-mode tangents of the flux of the conservative state
    double s[3], q[NV3_MAX], B[5][5], u[5];
    face_vector(p, a, i, j, k, s);
    const int c = cell_index(p, i, j, k);
    prim_at(p, U, c, q);
    coupling5_closed(q, s[0], s[1], s[2], lam, p.P.gamma, B);
    for (int v = 0; v < 5; ++v) u[v] = U[(size_t)v * p.NI * p.NJ * p.NK + c];
    for (int col = 0; col < 5; ++col) {
      Dual Ud[5], qd[5], F[5];
      for (int v = 0; v < 5; ++v) Ud[v] = Dual{u[v], v == col ? 1.0 : 0.0};
      to_prim3(Ud, qd, 5, p.P.gamma);
      normal_flux3(qd, s, p.P.gamma, F);
      for (int r = 0; r < 5; ++r) {
        const double ref = 0.5 * F[r].d - (r == col ? 0.5 * lam : 0.0);
        jworst = std::fmax(jworst, std::fabs(ref - B[r][col]));
        jscale = std::fmax(jscale, std::fabs(ref));
      }
    }
  }
  out[0] = worst / scale;
  out[1] = jworst / jscale;
  return 0;
}

// The Newton step's vector operations as host loops (sums in index order).
struct HostOps {
  enum { R_ = 0, Z_, W_, T_, RES_, B_, DU_, ACT_, BASE };
  const Plan3Dev& p;
  size_t N, n;
  std::vector<std::vector<double>> vec;
  std::vector<double> vdt;
  Linearised lin;
  HostOps(const Plan3Dev& plan, int m) : p(plan) {
    n = (size_t)p.NI * p.NJ * p.NK;
    N = (size_t)p.nvar * n;
    vec.assign(BASE + m + 1, std::vector<double>(N, 0.0));
    vdt.assign(n, 0.0);
  }
  int V(int i) const { return BASE + i; }
  double* d(int id) { return vec[id].data(); }
  void prepare(const double* U, double cfl) {
    LineTerms t;
    if (p.nvar > 5) line_terms<true>(p, U, cfl, t);
    else line_terms<false>(p, U, cfl, t);
    for (size_t c = 0; c < n; ++c) vdt[c] = t.sum[c] / cfl;
    linearise_as(p, U, lin);
  }
  void residual(const double* U, int out) { eval(p, U, nullptr, d(out), 0, false); }
  void matvec(const double* U, double, int src, int out) {
    lin_jv_as(p, lin, U, d(src), d(out));
    for (size_t e = 0; e < N; ++e) d(out)[e] = vdt[e % n] * d(src)[e] + d(out)[e];
  }
  void precondition(const double* U, double cfl, int src, int dst) { line_solve_as(p, U, cfl, d(src), d(dst)); }
  double dot(int a, int b) {
    double s = 0.0;
    for (size_t e = 0; e < N; ++e) s += d(a)[e] * d(b)[e];
    return s;
  }
  double nrm2(int a) { return std::sqrt(dot(a, a)); }
  void axpy(double al, int x, int y) { for (size_t e = 0; e < N; ++e) d(y)[e] = d(y)[e] + al * d(x)[e]; }
  void scale(double al, int x, int y) { for (size_t e = 0; e < N; ++e) d(y)[e] = al * d(x)[e]; }
  void copy(int x, int y) { vec[y] = vec[x]; }
  void zero(int y) { std::fill(vec[y].begin(), vec[y].end(), 0.0); }
  double density_norm(int r) {
    double a = 0.0, w = 0.0;
    for (size_t c = 0; c < n; ++c)
      if (p.interior[c]) {
        a += p.volume[c] * d(r)[c] * d(r)[c];
        w += p.volume[c];
      }
    return std::sqrt(a / w);
  }
  double worst_ratio(const double* U, int du) {
    double worst = 0.0;
    for (size_t c = 0; c < n; ++c) {
      double q[NV3_MAX];
      prim_at(p, U, (int)c, q);
      const double* D = d(du);
      double de = D[4 * n + c];
      for (int k = 0; k < 3; ++k) de = de - q[1 + k] * D[(1 + k) * n + c];
      const double vv = (q[1] * q[1] + q[2] * q[2]) + q[3] * q[3];
      const double dp = (p.P.gamma - 1.0) * (de + 0.5 * vv * D[c]);
      worst = std::fmax(worst, std::fabs(D[c]) / q[0]);
      worst = std::fmax(worst, std::fabs(dp) / q[4]);
      if (p.nvar > 5) {
        const double nh = U[5 * n + c] / q[0];
        const double dnh = (D[5 * n + c] - nh * D[c]) / q[0];
        worst = std::fmax(worst, std::fabs(dnh) / std::fmax(std::fabs(nh), 1.0));
      }
    }
    return worst;
  }
  bool physical_after(const double* U, int du) {
    std::vector<double> cand(N);
    for (size_t e = 0; e < N; ++e) {
      if (!std::isfinite(d(du)[e])) return false;
      cand[e] = U[e] + d(du)[e];
    }
    for (size_t c = 0; c < n; ++c) {
      double q[NV3_MAX];
      prim_at(p, cand.data(), (int)c, q);
      if (!(q[0] > 1e-10) || !(q[4] > 1e-10) || !std::isfinite(q[0]) || !std::isfinite(q[4])) return false;
    }
    return true;
  }
  void add_to_state(double* U, int du) { for (size_t e = 0; e < N; ++e) U[e] = U[e] + d(du)[e]; }
};

// Restarted GMRES over those operations (newton3d.cu's algorithm; the device keeps an Arnoldi
// step's scalars): (V/dt + J) X = B, ACTION = A X
static int gmres3(HostOps& ops, const double* U, double cfl, const Newton3Config& c, int B, int X, int ACTION) {
  const double tiny = 2.2250738585072014e-308;
  const double rcond = 2.220446049250313e-16 * (c.restart + 1);
  const int m = c.restart;
  auto prec = [&](int src, int dst) {
    if (c.preconditioner >= 1) ops.precondition(U, cfl, src, dst);
    else ops.copy(src, dst);
  };
  auto mdot = [&](int count, std::vector<double>& h) {
    for (int i = 0; i < count; ++i) h[i] = ops.dot(ops.V(i), HostOps::W_);
  };
  auto maxpy = [&](int count, const std::vector<double>& coef, int y) {
    for (int i = 0; i < count; ++i) ops.axpy(coef[i], ops.V(i), y);
  };
  const double bn = ops.nrm2(B);
  ops.zero(X);
  ops.copy(B, HostOps::R_);
  ops.zero(ACTION);
  std::vector<double> H((size_t)(m + 1) * m), h(m + 1), h2(m + 1), neg(m + 1), y, Hy(m + 1);
  for (int k = 0; k < c.maxiter; ++k) {
    const double rn = ops.nrm2(HostOps::R_);
    if (!(rn > c.tol * bn)) break;
    const double beta = rn;
    ops.scale(1.0 / std::fmax(beta, tiny), HostOps::R_, ops.V(0));
    std::fill(H.begin(), H.end(), 0.0);
    for (int j = 0; j < m; ++j) {
      prec(ops.V(j), HostOps::Z_);
      ops.matvec(U, cfl, HostOps::Z_, HostOps::W_);
      mdot(j + 1, h);
      for (int i = 0; i <= j; ++i) neg[i] = -h[i];
      maxpy(j + 1, neg, HostOps::W_);
      mdot(j + 1, h2);
      for (int i = 0; i <= j; ++i) neg[i] = -h2[i];
      maxpy(j + 1, neg, HostOps::W_);
      const double nrm = ops.nrm2(HostOps::W_);
      for (int i = 0; i <= j; ++i) H[(size_t)i * m + j] = h[i] + h2[i];
      H[(size_t)(j + 1) * m + j] = nrm;
      ops.scale(1.0 / std::fmax(nrm, tiny), HostOps::W_, ops.V(j + 1));
    }
    givens_lstsq(H, m, beta, rcond, y);
    ops.zero(HostOps::T_);
    maxpy(m, y, HostOps::T_);
    prec(HostOps::T_, HostOps::Z_);
    ops.axpy(1.0, HostOps::Z_, X);
    for (int i = 0; i <= m; ++i) {
      double s = 0.0;
      for (int j = 0; j < m; ++j) s = s + H[(size_t)i * m + j] * y[j];
      Hy[i] = s;
    }
    maxpy(m + 1, Hy, ACTION);
    ops.copy(B, HostOps::R_);
    ops.axpy(-1.0, ACTION, HostOps::R_);
  }
  return 0;
}

extern "C" int jr3_host_newton_steps(const jr_plan3d_desc* d, const double* config, const int* iconfig, double* U,
                                     double* cfl, double* res_prev, int n_steps, double* history) {
  HostPlan h;
  plan_of(d, h);
  Newton3Config c{iconfig[0], iconfig[1], iconfig[2], config[0], config[1], config[2], config[3], config[4],
                  config[5], config[6]};
  HostOps ops(h.p, c.restart);
  for (int s = 0; s < n_steps; ++s) history[s] = newton_step3(ops, U, *cfl, *res_prev, c);
  return 0;
}

// the 7 loads of every wall face (n_walls x 7) from the ghost-filled state
extern "C" int jr3_host_wall_loads(const jr_plan3d_desc* d, const double* U, double* loads) {
  HostPlan h;
  plan_of(d, h);
  const Plan3Dev& p = h.p;
  const std::vector<double> A = canvas<double>(p, U, nullptr);
  for (int w = 0; w < p.n_walls; ++w) wall_load(p, A.data(), w, loads + (size_t)7 * w);
  return 0;
}

extern "C" int jr3_host_forces(const jr_plan3d_desc* d, const double* U, double area, double length,
                               const double* centre, double* out) {
  std::vector<double> loads((size_t)d->n_walls * 7);
  jr3_host_wall_loads(d, U, loads.data());
  Physics3 P;
  physics3_from_desc(P, d);
  force_coefficients3(P, d->n_walls, loads.data(), d->wall_mid, area, length, centre, out);
  return 0;
}

// the wall distance of points (n x 3) to faces (m x 4 x 3), faces offered in order as the
// kernel offers them (bounded = 1: skipping by the bounding spheres; 0: every face ranked)
extern "C" int jr3_host_wall_distance(const double* points, long long n, const double* faces, int m, double* out,
                                      int bounded) {
  std::vector<double> spheres((size_t)4 * m);
  for (int f = 0; f < m; ++f) face_sphere(faces + (size_t)12 * f, spheres.data() + (size_t)4 * f);
  for (long long i = 0; i < n; ++i) {
    const V3 p = v3(points + 3 * i);
    Candidates c;
    c.init(m);
    for (int f = 0; f < m; ++f) {
      if (bounded) offer_face(c, p, faces + (size_t)12 * f, spheres.data() + (size_t)4 * f, f);
      else c.offer(face_rank_distance(p, faces + (size_t)12 * f), f);
    }
    out[i] = m > 0 ? candidates_distance(p, c, faces) : INFINITY;
  }
  return 0;
}

// the ghost-filled primitive canvas (nvar x canvas) at U: each ghost by its program, as the device
// fills it (mode 0), or by the stages, double-buffered (mode 1)
extern "C" int jr3_host_fill(const jr_plan3d_desc* d, const double* U, double* Q, int mode) {
  HostPlan h;
  plan_of(d, h);
  std::vector<double> A;
  if (mode == 0) {
    A = canvas<double>(h.p, U, nullptr);
  } else {
    std::vector<int> none(h.ghost_of.size(), -1);
    Plan3Dev own = h.p;
    own.ghost_of = none.data();
    A = canvas<double>(own, U, nullptr);
    fill_staged(h.p, d, A);
  }
  std::copy(A.begin(), A.end(), Q);
  return 0;
}
