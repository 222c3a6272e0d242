// The 3D wave speeds and line preconditioner kernels (bodies and layout in linesolve3d.cuh).
#include "linesolve3d.cuh"

namespace jr {

__global__ void k3_wave_speeds(Plan3Dev p, const double* __restrict__ U, double* __restrict__ lam) {
  const int n0 = face_count(p, 0), n1 = face_count(p, 1), n2 = face_count(p, 2);
  const int total = n0 + n1 + n2;
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < total; f += gridDim.x * blockDim.x) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    lam[f] = wave_speed(p, U, a, i, j, k);
  }
}

template <bool SA>
__global__ void __launch_bounds__(128) k3_line_faces(Plan3Dev p, const double* __restrict__ U, double* __restrict__ lam,
                                                     double* __restrict__ mflux, double* __restrict__ dflux, int nf) {
  for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
    int a, i, j, k;
    face_of(p, f, a, i, j, k);
    double l, m = 0.0, d = 0.0;
    line_face_terms<SA>(p, U, a, i, j, k, l, m, d);
    lam[f] = l;
    if constexpr (SA) {
      mflux[f] = m;
      dflux[f] = d;
    }
  }
}

// V/dt on every cell, and where chains run (block cells) their diagonals
template <bool SA>
__global__ void __launch_bounds__(128) k3_line_cells(Plan3Dev p, const double* __restrict__ U,
                                                     const double* __restrict__ lam, const double* __restrict__ mflux,
                                                     const double* __restrict__ dflux, double cfl,
                                                     double* __restrict__ dflow, double* __restrict__ dsa,
                                                     double* __restrict__ vdt) {
  const int n = p.NI * p.NJ * p.NK;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    double sum, d = 0.0;
    line_cell_terms<SA>(p, U, lam, mflux, dflux, cfl, c, sum, d);
    if (vdt != nullptr) vdt[c] = sum / cfl;
    dflow[c] = sum * (1.0 / cfl + 0.5);
    if constexpr (SA) dsa[c] = d;
  }
}

// line_factor_chain, one thread a chain: a step is
// a serial chain of five pivots, so its neighbours' chains are what hides it; its rows leave
// eight at a time, a sector a chain and word.  61,440 chains of 64: 1.1 ms, and the faces' and
// cells' terms 1.0 ms (assembling the blocks, every wave speed of a cell twice among them,
// as the one thread walked its chain: 16.2 ms).
template <class TF, bool SA>
__global__ void __launch_bounds__(64) k3_line_factor(Plan3Dev p, const double* __restrict__ U,
                                                     const double* __restrict__ lam, const double* __restrict__ mflux,
                                                     const double* __restrict__ dflux,
                                                     const double* __restrict__ dflow,
                                                     const double* __restrict__ dsa, TF* __restrict__ F) {
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch < p.n_chains) line_factor_chain<TF, SA>(p, U, lam, mflux, dflux, dflow, dsa, F, ch);
}

// z = M^-1 (s r) from the factor, s = *scale (1 where null); with vout the scaled input is also
// written there (a normalised Krylov vector).  Four chains a warp, eight lanes a chain: lane
// `row` holds its row's words and the vector's entry, the other rows' entries come by
// shuffles, and the words of the two elements ahead are in flight.  Bound by the factor's
// bytes where many chains run, by the sweeps' latency where few do: 61,440 coupled FP32 chains
// of 64, 638 us back to back, 0.80 ms in a step under the power cap (one thread a chain and a copy
// of the whole vector first: 1.14 ms); 3,072
// FP64 chains of 16, 21 us (231 us).  The blocks after the chains' copy the cells on no chain.
constexpr int LA_THREADS = 128, LA_CHAINS = LA_THREADS / 32 * LW_CHAINS;

template <class TF, int NV>
__global__ void __launch_bounds__(LA_THREADS) k3_line_apply(Plan3Dev p, const TF* __restrict__ F,
                                                            const double* __restrict__ r, double* __restrict__ z,
                                                            const double* __restrict__ scale,
                                                            double* __restrict__ vout, int chain_blocks) {
  const size_t n = (size_t)p.NI * p.NJ * p.NK;
  const double s = scale != nullptr ? *scale : 1.0;
  if ((int)blockIdx.x >= chain_blocks) {
    const size_t total = (size_t)p.n_offchain * NV, step = (size_t)(gridDim.x - chain_blocks) * LA_THREADS;
    for (size_t e = (size_t)(blockIdx.x - chain_blocks) * LA_THREADS + threadIdx.x; e < total; e += step) {
      const size_t at = e / p.n_offchain * n + p.offchain[e % p.n_offchain];
      const double x = s * r[at];
      z[at] = x;
      if (vout != nullptr) vout[at] = x;
    }
    return;
  }
  const int lane = threadIdx.x & 31, row = lane & 7, base = lane & 24;
  const int group = blockIdx.x * (LA_THREADS / 32) + threadIdx.x / 32, groups = line_groups(p), nc = p.n_chains;
  if (group >= groups) return;   // whole warps
  const int ch = group * LW_CHAINS + (lane >> 3);
  const bool mine = ch < nc && row < NV;
  const int len = ch < nc ? p.ch_len[ch] : 0;
  int most = len;
  most = max(most, __shfl_xor_sync(0xffffffffu, most, 8));
  most = max(most, __shfl_xor_sync(0xffffffffu, most, 16));
  const bool sa = NV > 5 && row == 5, coupled = NV > 5 && p.line_coupled;
  const size_t kstride = (size_t)groups * LW_WORDS * 32;
  const TF* Fw = F + (size_t)group * LW_WORDS * 32 + lane;
  const size_t ro = (size_t)row * n;
  constexpr int D = 2;   // elements in flight
  // 1. down: d_k = P_k (r_k - lower_k d_{k-1}); the uncoupled SA row beside the mean flow's
  {
    TF w[D][10];
    double rv[D];
    int cell[D];
    auto fetch = [&](int k, int b) {
      const bool in = mine && k < len;
      cell[b] = in ? p.ch_cells[(size_t)ch * p.chain_L + k] : -1;
      rv[b] = in ? r[ro + cell[b]] : 0.0;
      const TF* f = Fw + (size_t)k * kstride;
#pragma unroll
      for (int t = 0; t < 10; ++t) w[b][t] = in ? f[t * 32] : TF(0);
    };
#pragma unroll
    for (int b = 0; b < D; ++b)
      if (b < most) fetch(b, b);
    TF d = TF(0);
    for (int k0 = 0; k0 < most; k0 += D) {
#pragma unroll
      for (int b = 0; b < D; ++b) {
        const int k = k0 + b;
        if (k >= most) break;
        const double x = s * rv[b];
        const TF mr = TF(x);
        TF rhs, dn;
        {
          TF m = w[b][0] * __shfl_sync(0xffffffffu, d, base);
#pragma unroll
          for (int t = 1; t < 5; ++t) m = m + w[b][t] * __shfl_sync(0xffffffffu, d, base + t);
          rhs = mr - m;
          dn = w[b][5] * __shfl_sync(0xffffffffu, rhs, base);
#pragma unroll
          for (int t = 1; t < 5; ++t) dn = dn + w[b][5 + t] * __shfl_sync(0xffffffffu, rhs, base + t);
        }
        if (sa) dn = w[b][1] * (mr - w[b][0] * d);
        if (cell[b] >= 0) {
          if (!(coupled && sa)) {   // (the coupled SA row starts on the way back)
            d = dn;
            z[ro + cell[b]] = double(dn);
          }
          if (vout != nullptr) vout[ro + cell[b]] = x;
        }
        if (k + D < most) fetch(k + D, b);
      }
    }
  }
  // 2. back: x_k = d_k - C_k x_{k+1}.  Coupled, the SA row's right-hand side of element k + 1,
  // r - (lo x_k + up x_{k+2}), is complete once x_k is, and the SA chain's first sweep,
  // d_{k+1} = pivot (that - upper d_{k+2}), goes one element behind.
  {
    TF w[D][5];
    double dv[D];
    int cell[D];
    auto fetch = [&](int k, int b) {
      const bool in = ch < nc && k < len, vec = in && row < NV;
      cell[b] = vec ? p.ch_cells[(size_t)ch * p.chain_L + k] : -1;
      dv[b] = !vec ? 0.0 : (coupled && sa ? s * r[ro + cell[b]] : z[ro + cell[b]]);
      const TF* f = Fw + (size_t)k * kstride;
#pragma unroll
      for (int t = 0; t < 5; ++t) w[b][t] = in && (row < NV || coupled) ? f[(10 + t) * 32] : TF(0);
    };
#pragma unroll
    for (int b = 0; b < D; ++b)
      if (most - 1 - b >= 0) fetch(most - 1 - b, b);
    TF x = TF(0);
    // of element k + 1: its coupling words (row 6), up x_{k+2} (row 7); the SA lane's r, upper,
    // pivot and cell
    TF pw[5] = {}, pup = TF(0), pr = TF(0), pupper = TF(0), ppiv = TF(0);
    int pcell = -1;
    auto finish = [&](TF lo) {   // the SA row's element k + 1
      const TF lo_all = __shfl_sync(0xffffffffu, lo, base + 6), up_all = __shfl_sync(0xffffffffu, pup, base + 7);
      if (sa && pcell >= 0) {
        x = ppiv * ((pr - (lo_all + up_all)) - pupper * x);
        z[ro + pcell] = double(x);
      }
    };
    for (int k0 = most - 1; k0 >= 0; k0 -= D) {
#pragma unroll
      for (int b = 0; b < D; ++b) {
        const int k = k0 - b;
        if (k < 0) break;
        TF xt[5];   // the mean flow's x_{k+1}
#pragma unroll
        for (int t = 0; t < 5; ++t) xt[t] = __shfl_sync(0xffffffffu, x, base + t);
        TF m = w[b][0] * (sa ? x : xt[0]);
        if (!sa)
#pragma unroll
          for (int t = 1; t < 5; ++t) m = m + w[b][t] * xt[t];
        if (cell[b] >= 0 && !(coupled && sa)) {
          x = TF(dv[b]) - m;
          z[ro + cell[b]] = double(x);
        }
        if (coupled) {
          TF lo = pw[0] * __shfl_sync(0xffffffffu, x, base);
#pragma unroll
          for (int t = 1; t < 5; ++t) lo = lo + pw[t] * __shfl_sync(0xffffffffu, x, base + t);
          finish(lo);
          pup = k + 1 < len ? m : TF(0);   // row 7: its words are the coupling above
#pragma unroll
          for (int t = 0; t < 5; ++t) pw[t] = w[b][t];
          pr = TF(dv[b]);
          pupper = w[b][0];
          ppiv = w[b][1];
          pcell = cell[b];
        }
        if (k - D >= 0) fetch(k - D, b);
      }
    }
    if (coupled) finish(TF(0));   // element 0 has nothing below
  }
  if (!coupled || !sa || ch >= nc) return;
  // 3. coupled: the SA row forward, x_k = d_k - c_k x_{k-1}
  {
    const TF* plane = F + line_words(p) + ch;
    const size_t pstride = (size_t)groups * LW_CHAINS;
    constexpr int DS = 4;
    TF x = TF(0), wc[DS];
    double dv[DS];
    int cell[DS];
    auto fetch = [&](int k, int b) {
      cell[b] = p.ch_cells[(size_t)ch * p.chain_L + k];
      dv[b] = z[ro + cell[b]];
      wc[b] = plane[(size_t)k * pstride];
    };
#pragma unroll
    for (int b = 0; b < DS; ++b)
      if (b < len) fetch(b, b);
    for (int k0 = 0; k0 < len; k0 += DS)
#pragma unroll
      for (int b = 0; b < DS; ++b) {
        const int k = k0 + b;
        if (k >= len) break;
        x = TF(dv[b]) - wc[b] * x;
        z[ro + cell[b]] = double(x);
        if (k + DS < len) fetch(k + DS, b);
      }
  }
}

void launch_wave_speeds3(const Plan3Dev& p, const double* U, double* lam, cudaStream_t st) {
  const int total = face_count(p, 0) + face_count(p, 1) + face_count(p, 2);
  counted3();
  k3_wave_speeds<<<(total + 127) / 128, 128, 0, st>>>(p, U, lam);
}

size_t line_factor_words3(const Plan3Dev& p) {
  return line_words(p) + (size_t)p.chain_L * line_groups(p) * LW_CHAINS;
}

template <class TF, bool SA>
static void factor_chains(const Plan3Dev& p, const double* U, const double* lam, const double* m, const double* d,
                          const double* dflow, const double* dsa, void* F, cudaStream_t st) {
  k3_line_factor<TF, SA><<<(p.n_chains + 63) / 64, 64, 0, st>>>(p, U, lam, m, d, dflow, dsa, static_cast<TF*>(F));
}

// V/dt at (U, cfl) into vdt (may be null) and, where F is given, the line_j factor into F
// (line_factor_words3 words, FP32 where p.line_fp32, else FP64).  The faces' and cells' terms
// stay in p.face_buf between the launches (planes of all faces: lambda, the SA mass flux and
// diffusion, then the cells' two diagonals), which the residual overwrites.
void launch_line_factor3(const Plan3Dev& p, const double* U, double cfl, void* F, double* vdt, cudaStream_t st) {
  const int nf = face_count(p, 0) + face_count(p, 1) + face_count(p, 2), n = p.NI * p.NJ * p.NK;
  double *lam = p.face_buf, *m = lam + nf, *d = m + nf, *dflow = d + nf, *dsa = dflow + nf;
  const bool sa = p.nvar > 5;
  counted3(2);
  if (sa) {
    k3_line_faces<true><<<(nf + 127) / 128, 128, 0, st>>>(p, U, lam, m, d, nf);
    k3_line_cells<true><<<(n + 127) / 128, 128, 0, st>>>(p, U, lam, m, d, cfl, dflow, dsa, vdt);
  } else {
    k3_line_faces<false><<<(nf + 127) / 128, 128, 0, st>>>(p, U, lam, m, d, nf);
    k3_line_cells<false><<<(n + 127) / 128, 128, 0, st>>>(p, U, lam, m, d, cfl, dflow, dsa, vdt);
  }
  if (F == nullptr || p.n_chains == 0) return;
  counted3();
  if (p.line_fp32) {
    if (sa) factor_chains<float, true>(p, U, lam, m, d, dflow, dsa, F, st);
    else factor_chains<float, false>(p, U, lam, m, d, dflow, dsa, F, st);
  } else {
    if (sa) factor_chains<double, true>(p, U, lam, m, d, dflow, dsa, F, st);
    else factor_chains<double, false>(p, U, lam, m, d, dflow, dsa, F, st);
  }
}

// z = M^-1 (*scale r) from the factor F (scale null: 1), cells on no chain copied; vout (may
// be null) receives *scale r
void launch_line_apply3(const Plan3Dev& p, const void* F, const double* r, double* z, const double* scale, double* vout,
                        cudaStream_t st) {
  const int chains = (p.n_chains + LA_CHAINS - 1) / LA_CHAINS;
  const int copies = (int)((size_t)p.n_offchain * p.nvar / 1024 + 1);
  const unsigned grid = (unsigned)(chains + (copies < 1184 ? copies : 1184));
  counted3();
  if (p.line_fp32) {
    const float* f = static_cast<const float*>(F);
    if (p.nvar > 5) k3_line_apply<float, 6><<<grid, LA_THREADS, 0, st>>>(p, f, r, z, scale, vout, chains);
    else k3_line_apply<float, 5><<<grid, LA_THREADS, 0, st>>>(p, f, r, z, scale, vout, chains);
  } else {
    const double* f = static_cast<const double*>(F);
    if (p.nvar > 5) k3_line_apply<double, 6><<<grid, LA_THREADS, 0, st>>>(p, f, r, z, scale, vout, chains);
    else k3_line_apply<double, 5><<<grid, LA_THREADS, 0, st>>>(p, f, r, z, scale, vout, chains);
  }
}

void launch_precondition3(const Plan3Dev& p, const double* U, double cfl, const double* r, double* z, void* F,
                          cudaStream_t st) {
  launch_line_factor3(p, U, cfl, F, nullptr, st);
  launch_line_apply3(p, F, r, z, nullptr, nullptr, st);
}

}  // namespace jr
