// Right-preconditioned restarted GMRES (src/jaxrans/solvers/krylov.py:34-137) and the
// pseudo-transient Newton update (src/jaxrans/solvers/implicit.py:54-168), on the device.
//
// Every cycle runs with a fixed launch sequence (so a Newton step can be captured in
// one CUDA graph): the kernels of a cycle read the case's `active` flag and return at
// once when the restart loop has already stopped.  CGS2 is three reads of the basis:
// the dots; the first update fused with the second dots; the second update fused with
// the norm.  Reductions are per-block partial sums finished by the last block in a fixed
// order, so a rerun gives bitwise the same scalars.  TV is the basis type (double;
// float in the mixed form, with FP64 accumulation).
#include "device.cuh"
#include "orth.cuh"

namespace jr {

constexpr int RED_THREADS = 256;

__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}

// NaN-propagating max
__device__ __forceinline__ double nmax(double a, double b) { return (a != a || b != b) ? NAN : (a > b ? a : b); }

__device__ __forceinline__ double warp_max(double x) {
  for (int o = 16; o > 0; o >>= 1) x = nmax(x, __shfl_down_sync(0xffffffffu, x, o));
  return x;
}

// In the last block of a reduction: out[k] = the sum (or NaN-propagating max) over the
// nb rows of partial[b * stride + k], k < W, by all the block's threads in a fixed order
// -- thread (k, r) takes the rows b = r, r + R, ... (R = blockDim.x / W groups), with its
// loads issued eight at a time, then the R group totals are added by halves.  Loads go
// to L2 (ld.global.cg), where the other blocks' partials are.
template <bool MAX>
__device__ void reduce_rows(const double* partial, int stride, int W, int nb, double* out) {
  __shared__ double group[RED_THREADS];
  const int R = max(1, (int)blockDim.x / W);
  const int t = threadIdx.x, k = t % W, r = t / W;
  if (r < R) {
    double acc = MAX ? -INFINITY : 0.0;
    // rows r, r + R, ... in order, eight loads in flight at a time (the last eight
    // predicated, so the tail costs one round trip, not one per row)
    for (int b = r; b < nb; b += 8 * R) {
      double x[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) x[u] = b + u * R < nb ? __ldcg(partial + (size_t)(b + u * R) * stride + k) : 0.0;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (b + u * R < nb) acc = MAX ? nmax(acc, x[u]) : acc + x[u];
    }
    group[t] = acc;
  }
  __syncthreads();
  // the R groups by halving (one after another they are a serial chain of R shared loads)
  int half = 1;
  while (2 * half < R) half *= 2;
  for (; half > 0; half >>= 1) {
    if (r < half && r + half < R) group[t] = MAX ? nmax(group[t], group[t + half * W]) : group[t] + group[t + half * W];
    __syncthreads();
  }
  if (t < W) out[t] = group[t];
  __syncthreads();
}

// Block-sums `vals` into partial[block * W + k]; true in thread 0 of the last block to
// finish, whose `vals` then hold the fixed-order totals over blocks.
template <int W, bool MAX = false>
__device__ bool reduce_last(double (&vals)[W], double* partial, unsigned* ticket, int nb) {
  __shared__ double sm[RED_THREADS / 32][W];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    double x = MAX ? warp_max(vals[k]) : warp_sum(vals[k]);
    if (lane == 0) sm[warp][k] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < W; ++k) {
      double t = sm[0][k];
      for (int w = 1; w < nw; ++w) t = MAX ? nmax(t, sm[w][k]) : t + sm[w][k];
      partial[blockIdx.x * W + k] = t;
    }
    __threadfence();
    unsigned prev = atomicAdd(ticket, 1u);
    last = prev == (unsigned)nb - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  __shared__ double total[W];
  reduce_rows<MAX>(partial, W, W, nb, total);
  if (threadIdx.x != 0) return false;
#pragma unroll
  for (int k = 0; k < W; ++k) vals[k] = total[k];
  *ticket = 0u;
  return true;
}

// The range of elements block b of nb owns
__device__ __forceinline__ void chunk(int n, int nb, int& lo, int& hi) {
  int per = (n + nb - 1) / nb;
  lo = blockIdx.x * per;
  hi = min(n, lo + per);
}

// ---- GMRES ---------------------------------------------------------------------------
// Every kernel takes the batch's case table and reads its case from blockIdx.y.  The
// per-case block count of a reduction depends on that case's size alone, so a case's
// scalars are bitwise the same alone and in a batch; the blocks past it return at once.

// blocks of a chunked per-case reduction over n elements (<= the grid's x)
__device__ __forceinline__ bool chunk_owner(int n, int& nb, int& lo, int& hi) {
  nb = chunk_blocks(n);
  if ((int)blockIdx.x >= nb) return false;
  chunk(n, nb, lo, hi);
  return true;
}

// Start of a Newton step: b = -R, x = action = 0, r = b; |b|; the residual norm of the
// density row from the tile partials; the history entry.
__global__ void __launch_bounds__(RED_THREADS) k_gmres_init(const CaseDev* __restrict__ cases, int n_cases_hist) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  const int n = cd.n_vec;
  int nb, lo, hi;
  if (!chunk_owner(n, nb, lo, hi)) return;
  const double* __restrict__ R = cd.R;
  double *b = cd.b, *r = cd.r, *x = cd.x, *action = cd.action;
  double acc[1] = {0.0};
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    double v = -R[i];
    b[i] = v;
    r[i] = v;
    x[i] = 0.0;
    action[i] = 0.0;
    acc[0] += v * v;
  }
  if (blockIdx.x == 0) {   // the residual's norm, from its tiles' sums by all the block's threads
    __shared__ double total;
    reduce_rows<false>(cd.tile_partial, 1, 1, cd.n_tiles, &total);
    if (threadIdx.x == 0) {
      Scalars* sc = cd.sc;
      const double nrm = sqrt(total / cd.c.volume_sum);
      sc->norm = nrm;
      // history: [step][case] over the cases of the batch
      if (cd.history != nullptr) cd.history[(size_t)sc->hpos * n_cases_hist + cd.slot] = nrm;
      sc->hpos += 1;
    }
  }
  if (reduce_last<1>(acc, cd.partial, cd.ticket, nb)) {
    Scalars* sc = cd.sc;
    sc->bnorm = sqrt(acc[0]);
    sc->rnorm = sc->bnorm;
    sc->cycle = 0;
    sc->active = 1;
    sc->status &= ST_STAGE_FAILED;
  }
}

// Cycle start: the restart test between cycles, beta = |r|; H = 0
__global__ void k_cycle_start(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  const Config& cfg = cd.cfg;
  for (int k = threadIdx.x; k < (cfg.restart + 1) * cfg.restart; k += blockDim.x) sc->H[k] = 0.0;
  if (threadIdx.x != 0) return;
  bool go = sc->active != 0 && sc->cycle < cfg.maxiter && sc->rnorm > cfg.krylov_tol * sc->bnorm;
  sc->active = go ? 1 : 0;
  sc->beta = sc->rnorm;
  sc->inv_nrm = 1.0 / fmax(sc->beta, 2.2250738585072014e-308);
}

// The gate of a Krylov cycle in the step graph: the cycle's body (an IF node) runs only
// when some case of the launch is still active; `cycles` counts the bodies run.
__global__ void k_cycle_gate(const CaseDev* __restrict__ cases, int n_cases, cudaGraphConditionalHandle gate,
                             unsigned long long* cycles) {
  int any = 0;
  for (int k = threadIdx.x; k < n_cases; k += blockDim.x) any |= cases[k].enabled && cases[k].sc->active != 0;
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    cudaGraphSetConditional(gate, any ? 1u : 0u);
    if (any) *cycles += 1ull;
  }
}

// The three passes of CGS2 over an FP64 basis: h1 = V^T w; w -= V h1, then h2 = V^T w; w -= V h2,
// then |w| and column j of H.  A block owns a contiguous part of a case (orth_blocks(n) of
// them, at most one an SM).  Two forms of the first two passes give the same bits: every dot
// product is a thread's elements in order, its warp's lanes by halves, the block's eight warps and
// the blocks in order.
//
// Few blocks (k_orth_dots): a thread holds its E elements' entries of every vector in registers,
// so the second pass updates w and takes its dots from one read of the basis, and NK x E loads a
// thread are in flight.  On one 385 x 97 case (194k unknowns) a pass is its latency: launch, a few
// rounds of loads, the sums' two stages; the three over 8, 15 and 30 vectors take 25, 29 and 37 us, on a
// 769 x 193 case 35, 58 and 134 us (a warp a vector, the second pass reading the basis twice: 29, 38 and
// 54 us; 45, 76 and 189 us).  E by those two cases: at one element a thread the 769 x 193 case takes 37
// and 65 us over 8 and 15 vectors, over 30 the same (two would spill; four of eight with the update
// spill 20 bytes).

// The dots of the NK vectors from k0 (nk of them) with w, after (UPDATE) w -= sum h V over the
// same vectors.  second: h1 in, h2 out; else h1 out.
template <int NK, int E, bool UPDATE>
__global__ void __launch_bounds__(ORTH_THREADS, NK <= 8 ? 2 : 1)
    k_orth_dots(const CaseDev* __restrict__ cases, int k0, int nk, int second) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int n = cd.n_vec, nb = orth_blocks(n);
  if ((int)blockIdx.x >= nb) return;
  const size_t ldv = (size_t)n;
  const double* __restrict__ V = (const double*)cd.V + (size_t)k0 * ldv;
  double* __restrict__ w = cd.w;
  double* hout = (second ? sc->h2 : sc->h1) + k0;
  __shared__ double h[NK], total[NK];
  if (UPDATE) {
    if ((int)threadIdx.x < NK) h[threadIdx.x] = (int)threadIdx.x < nk ? sc->h1[k0 + threadIdx.x] : 0.0;
    __syncthreads();
  }
  int lo, hi;
  chunk(n, nb, lo, hi);
  double acc[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) acc[k] = 0.0;
  for (int e = lo + threadIdx.x; e < hi; e += E * ORTH_THREADS) {
    double x[E];
    double v[E][NK];
#pragma unroll
    for (int i = 0; i < E; ++i) {
      const int at = e + i * ORTH_THREADS;
      x[i] = at < hi ? w[at] : 0.0;
#pragma unroll
      for (int k = 0; k < NK; ++k) v[i][k] = k < nk && at < hi ? V[k * ldv + at] : 0.0;
    }
    if (UPDATE) {
#pragma unroll
      for (int i = 0; i < E; ++i) {
        const int at = e + i * ORTH_THREADS;
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NK; ++k)
          if (k < nk) s += h[k] * v[i][k];
        x[i] -= s;
        if (at < hi) w[at] = x[i];
      }
    }
#pragma unroll
    for (int k = 0; k < NK; ++k)
      if (k < nk)
#pragma unroll
        for (int i = 0; i < E; ++i) acc[k] += v[i][k] * x[i];
  }
  if (finish_sums<NK>(acc, cd.partial, cd.ticket, nb, total) && (int)threadIdx.x < nk)
    hout[threadIdx.x] = total[threadIdx.x];
}

// Many blocks, each with few elements (k_orth_dots_dense): in the form above one block is all an
// SM holds, so the blocks' loads and sums follow one another, and of a thread's work on two elements
// the sums over its warp are most.  Here w (updated, for UPDATE, from a first read of the
// block's part of the basis, which its dots then find in L1 or L2) lies in shared memory, and a warp
// takes a vector, its lanes the elements of all eight warps of the form above, a sum each: 9
// shuffles a vector in place of 31 for 32 sums in each of eight warps.  Four blocks an SM.
template <int NK, bool UPDATE>
__global__ void __launch_bounds__(ORTH_THREADS, 4)
    k_orth_dots_dense(const CaseDev* __restrict__ cases, int k0, int nk, int second) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int n = cd.n_vec, nb = orth_blocks(n);
  if ((int)blockIdx.x >= nb) return;
  const size_t ldv = (size_t)n;
  const double* __restrict__ V = (const double*)cd.V + (size_t)k0 * ldv;
  double* __restrict__ w = cd.w;
  double* hout = (second ? sc->h2 : sc->h1) + k0;
  extern __shared__ double ws[];   // the block's part of w, zeros to a whole round
  __shared__ double h[NK], total[NK];
  if (UPDATE) {
    if ((int)threadIdx.x < NK) h[threadIdx.x] = (int)threadIdx.x < nk ? sc->h1[k0 + threadIdx.x] : 0.0;
    __syncthreads();
  }
  int lo, hi;
  chunk(n, nb, lo, hi);
  const int len = hi - lo, padded = (len + ORTH_ROUND - 1) / ORTH_ROUND * ORTH_ROUND;
  for (int e = threadIdx.x; e < padded; e += ORTH_THREADS) {
    double x = 0.0;
    if (e < len) {
      x = w[lo + e];
      if (UPDATE) {
        constexpr int KB = 8;
        double s = 0.0;
#pragma unroll
        for (int b = 0; b < NK; b += KB) {
          double v[KB];
#pragma unroll
          for (int k = 0; k < KB; ++k) v[k] = V[(size_t)min(b + k, nk - 1) * ldv + lo + e];   // (no branch: all in flight)
#pragma unroll
          for (int k = 0; k < KB; ++k)
            if (b + k < nk) s += h[b + k] * v[k];
        }
        x -= s;
        w[lo + e] = x;
      }
    }
    ws[e] = x;
  }
  __syncthreads();
  constexpr int NW = ORTH_THREADS / 32, NV = ORTH_ROUND / 32;
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < nk; k += NW) {
    const double* __restrict__ vk = V + k * ldv + lo;
    double a[NW] = {};
    for (int e = lane; e < padded; e += ORTH_ROUND) {
      double v[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) v[q] = e + 32 * q < len ? vk[e + 32 * q] : 0.0;
#pragma unroll
      for (int q = 0; q < NV; ++q) a[q % NW] += v[q] * ws[e + 32 * q];
    }
    lane_sums<NW>(a, lane);
    double s = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
    for (int q = 1; q < NW; ++q) s += __shfl_sync(0xffffffffu, a[0], q * (32 / NW));
    if (lane == 0) cd.partial[(size_t)blockIdx.x * NK + k] = s;
  }
  if (finish_blocks<NK>(cd.partial, cd.ticket, nb, total) && (int)threadIdx.x < nk)
    hout[threadIdx.x] = total[threadIdx.x];
}

// w -= sum h V over all nk vectors (h: h2, or h1 where `first`), and with `column` |w| and
// column j of H.  Two elements a thread and 32 loads in flight where the blocks are few; DENSE: one
// element, eight loads, four blocks an SM (the same bits).
template <bool DENSE>
__global__ void __launch_bounds__(ORTH_THREADS, DENSE ? 4 : 2)
    k_orth_update(const CaseDev* __restrict__ cases, int nk, int j, int first, int column) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int n = cd.n_vec, m = cd.m, nb = orth_blocks(n);
  if ((int)blockIdx.x >= nb) return;
  const size_t ldv = (size_t)n;
  const double* __restrict__ V = (const double*)cd.V;
  double* __restrict__ w = cd.w;
  __shared__ double h[MAX_KRYLOV], total[8];
  if ((int)threadIdx.x < nk) h[threadIdx.x] = (first ? sc->h1 : sc->h2)[threadIdx.x];
  __syncthreads();
  int lo, hi;
  chunk(n, nb, lo, hi);
  double acc[8] = {};
  constexpr int E = DENSE ? 1 : 2, KB = DENSE ? 8 : 16;
  for (int e = lo + threadIdx.x; e < hi; e += E * ORTH_THREADS) {
    double x[E], s[E] = {};
#pragma unroll
    for (int i = 0; i < E; ++i) x[i] = e + i * ORTH_THREADS < hi ? w[e + i * ORTH_THREADS] : 0.0;
    for (int k0 = 0; k0 < nk; k0 += KB) {
      double v[E][KB];
#pragma unroll
      for (int i = 0; i < E; ++i)
#pragma unroll
        for (int k = 0; k < KB; ++k) {
          // (DENSE: the count alone would be a branch, and the loads after it wait; clamped, all are
          // in flight.  Two elements: the second's bound is a thread's own, so the loads are predicated)
          if constexpr (DENSE) v[i][k] = V[(size_t)min(k0 + k, nk - 1) * ldv + e];
          else v[i][k] = k0 + k < nk && e + i * ORTH_THREADS < hi ? V[(k0 + k) * ldv + e + i * ORTH_THREADS] : 0.0;
        }
#pragma unroll
      for (int k = 0; k < KB; ++k)
        if (k0 + k < nk)
#pragma unroll
          for (int i = 0; i < E; ++i) s[i] += h[k0 + k] * v[i][k];
    }
#pragma unroll
    for (int i = 0; i < E; ++i) {
      x[i] -= s[i];
      acc[0] += x[i] * x[i];
      if (e + i * ORTH_THREADS < hi) w[e + i * ORTH_THREADS] = x[i];
    }
  }
  if (!column || !finish_sums<8>(acc, cd.partial, cd.ticket, nb, total)) return;
  const double nrm = sqrt(total[0]);
  if ((int)threadIdx.x < nk) sc->H[threadIdx.x + (m + 1) * j] = sc->h1[threadIdx.x] + sc->h2[threadIdx.x];
  if (threadIdx.x == 0) {
    sc->H[j + 1 + (m + 1) * j] = nrm;
    sc->nrm = nrm;
    sc->inv_nrm = 1.0 / fmax(nrm, 2.2250738585072014e-308);
    if (nrm == 0.0) sc->status |= ST_GMRES_BREAKDOWN;
  }
}

// The same passes over an FP32 basis (the mixed form), one kernel: MODE 0, 1, 2.  A block owns a
// chunk of cgs_chunk(n) elements; the update runs thread per element and the dot products warp
// per basis vector against the block's w in shared memory, 16 loads in flight a lane, so the
// FP64 conversions follow whole batches of loads.  Holding the entries in registers as the
// FP64 passes do is slower here (the loads, each with its conversion, are not issued
// together): nine cases' 442k cells, three passes over 30 vectors, 324 against 488 us.
template <int NK, int MODE>
__global__ void __launch_bounds__(RED_THREADS) k_mdot_fp32(const CaseDev* __restrict__ cases, int nk, int j) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int n = cd.n_vec, m = cd.m;
  const int nb = cgs_blocks(n), C = cgs_chunk(n);
  if ((int)blockIdx.x >= nb) return;
  const float* __restrict__ V = (const float*)cd.V;
  const size_t ldv = (size_t)n;
  double* __restrict__ w = cd.w;
  double* __restrict__ partial = cd.partial;
  unsigned* ticket = cd.ticket;
  const double* hin = MODE == 1 ? sc->h1 : sc->h2;
  double* hout = MODE == 0 ? sc->h1 : sc->h2;
  __shared__ double ws[MODE == 2 ? 1 : CGS_MAX_CHUNK];
  __shared__ double h[MODE == 0 ? 1 : NK];
  __shared__ double sm[RED_THREADS / 32];
  __shared__ bool last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if constexpr (MODE != 0) {
    if ((int)threadIdx.x < NK) h[threadIdx.x] = (int)threadIdx.x < nk ? hin[threadIdx.x] : 0.0;
    __syncthreads();
  }
  const int i0 = blockIdx.x * C;
  const int cn = min(C, n - i0);
  // 1. the update (MODE 1, 2), or the copy of w (MODE 0), element by element
  double acc = 0.0;
  for (int e = threadIdx.x; e < cn; e += blockDim.x) {
    const int i = i0 + e;
    double wi = w[i];
    if constexpr (MODE != 0) {
      double s = 0.0;
      // The 16-vector kernels load under the count's branch, the others select what they loaded:
      // the same sums, but ptxas schedules the loads so differently that the branch takes the three
      // passes over 8 vectors 46 -> 50 us on a 769 x 193 case and over 30 vectors 106 -> 120, eight
      // 385 x 97 cases 219 -> 230, yet over 15 vectors 61 -> 57 and 138 -> 125.
      if constexpr (NK == 16) {
#pragma unroll
        for (int k = 0; k < NK; ++k)
          if (k < nk) s += h[k] * double(V[(size_t)k * ldv + i]);
      } else {
        constexpr int KB = 1;
#pragma unroll
        for (int k0 = 0; k0 < NK; k0 += KB) {
          double vk[KB];
#pragma unroll
          for (int u = 0; u < KB; ++u) vk[u] = k0 + u < nk ? double(V[(size_t)(k0 + u) * ldv + i]) : 0.0;
#pragma unroll
          for (int u = 0; u < KB; ++u)
            if (k0 + u < nk) s += h[k0 + u] * vk[u];
        }
      }
      wi = wi - s;
      w[i] = wi;
    }
    if constexpr (MODE == 2) acc += wi * wi;
    else ws[e] = wi;
  }
  const int width = MODE == 2 ? 1 : nk;
  if constexpr (MODE == 2) {
    double x = warp_sum(acc);
    if (lane == 0) sm[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = sm[0];
      for (int ww = 1; ww < nw; ++ww) t += sm[ww];
      partial[blockIdx.x * (MAX_KRYLOV + 1)] = t;
    }
  } else {
    __syncthreads();
    // 2. the dot products, warp per basis vector
    for (int k = warp; k < nk; k += nw) {
      const float* __restrict__ vk = V + k * ldv + i0;
      double a = 0.0;
      int e = lane;
      for (; e + 32 * 15 < cn; e += 32 * 16) {
        double x[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) x[u] = double(vk[e + 32 * u]);
#pragma unroll
        for (int u = 0; u < 16; ++u) a += x[u] * ws[e + 32 * u];
      }
      for (; e < cn; e += 32) a += double(vk[e]) * ws[e];
      a = warp_sum(a);
      if (lane == 0) partial[blockIdx.x * (MAX_KRYLOV + 1) + k] = a;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == (unsigned)nb - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double total[MAX_KRYLOV + 1];
  reduce_rows<false>(partial, MAX_KRYLOV + 1, width, nb, total);
  if ((int)threadIdx.x < width) {
    const double t = total[threadIdx.x];
    if constexpr (MODE == 2) {
      double nrm = sqrt(t);
      for (int k = 0; k < nk; ++k) sc->H[k + (m + 1) * j] = sc->h1[k] + sc->h2[k];
      sc->H[j + 1 + (m + 1) * j] = nrm;
      sc->nrm = nrm;
      sc->inv_nrm = 1.0 / fmax(nrm, 2.2250738585072014e-308);
      if (nrm == 0.0) sc->status |= ST_GMRES_BREAKDOWN;
    } else {
      hout[threadIdx.x] = t;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) *ticket = 0u;
}

// argmin |beta e1 - H y| by Givens rotations, pivots below rcond * the largest dropped
// (krylov.py:100-137); hy = H y.  One warp per case, columns over its lanes: rotation j, once
// formed by the lane that holds column j, is applied to rows j, j+1 of every later column at
// once -- each entry sees the same rotations in the same order as column-by-column
// elimination -- and the back substitution takes column j out of every row above at once.  A
// serial chain of m roots and quotients: no block barrier lies in it (m = 30: 32 us as two
// warps with three barriers a rotation, 20 us so; m = 10: 11 -> 7 us).
__global__ void __launch_bounds__(32) k_lstsq(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int m = cd.m, lane = threadIdx.x;
  __shared__ double h[MAX_KRYLOV + 1][MAX_KRYLOV + 1];
  __shared__ double g[MAX_KRYLOV + 1], y[MAX_KRYLOV];
  for (int e = lane; e < (m + 1) * m; e += 32) h[e % (m + 1)][e / (m + 1)] = sc->H[e];
  for (int i = lane; i <= m; i += 32) g[i] = i == 0 ? sc->beta : 0.0;
  __syncwarp();
  double largest = 0.0;
  for (int j = 0; j < m; ++j) {
    // every lane forms the rotation from the same two entries
    const double a = h[j][j], c = h[j + 1][j];
    const double r = sqrt(a * a + c * c);
    const double safe = r > 0.0 ? r : 1.0;
    const double cj = r > 0.0 ? a / safe : 1.0, sj = r > 0.0 ? c / safe : 0.0;
    const double gj = g[j];
    __syncwarp();
    largest = j == 0 ? r : fmax(largest, r);
    for (int col = j + 1 + lane; col < m; col += 32) {
      const double p = h[j][col], q = h[j + 1][col];
      h[j][col] = cj * p + sj * q;
      h[j + 1][col] = cj * q - sj * p;
    }
    if (lane == 0) {
      h[j][j] = r;
      h[j + 1][j] = 0.0;
      g[j] = cj * gj;
      g[j + 1] = -sj * gj;
    }
    __syncwarp();
  }
  const double rcond = 2.220446049250313e-16 * (m + 1);
  for (int j = m - 1; j >= 0; --j) {
    const double d = h[j][j];
    const double yj = fabs(d) > rcond * largest ? g[j] / d : 0.0;
    __syncwarp();
    for (int i = lane; i < j; i += 32) g[i] -= h[i][j] * yj;
    if (lane == 0) y[j] = yj;
    __syncwarp();
  }
  for (int i = lane; i < m; i += 32) sc->y[i] = y[i];
  for (int i = lane; i <= m; i += 32) {
    double s = 0.0;
#pragma unroll 8
    for (int jj = 0; jj < m; ++jj) s += sc->H[i + (m + 1) * jj] * y[jj];
    sc->hy[i] = s;
  }
}

// tmp = V_{0..m-1} y; action += V_{0..m} (H y), V_m = w / |w|
template <class TV>
__global__ void k_combine(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  const Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  const int m = cd.m, n = cd.n_vec;
  const TV* __restrict__ V = (const TV*)cd.V;
  const size_t ldv = (size_t)n;
  const double* __restrict__ w = cd.w;
  double* __restrict__ tmp = cd.tmp;
  double* __restrict__ action = cd.action;
  __shared__ double y[MAX_KRYLOV], hy[MAX_KRYLOV + 1];
  if ((int)threadIdx.x < m) y[threadIdx.x] = sc->y[threadIdx.x];
  if ((int)threadIdx.x <= m) hy[threadIdx.x] = sc->hy[threadIdx.x];
  __syncthreads();
  const double inv = sc->inv_nrm;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double s = 0.0, a = 0.0;
    for (int k = 0; k < m; ++k) {
      double v = double(V[k * ldv + i]);
      s += y[k] * v;
      a += hy[k] * v;
    }
    a += hy[m] * double(TV(w[i] * inv));
    tmp[i] = s;
    action[i] += a;
  }
}

// x += z; r = b - action; |r|; the cycle count
__global__ void __launch_bounds__(RED_THREADS) k_cycle_end(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  Scalars* sc = cd.sc;
  if (sc->active == 0) return;
  int nb, lo, hi;
  if (!chunk_owner(cd.n_vec, nb, lo, hi)) return;
  double *x = cd.x, *r = cd.r;
  const double *z = cd.z, *b = cd.b, *action = cd.action;
  double acc[1] = {0.0};
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    x[i] += z[i];
    double ri = b[i] - action[i];
    r[i] = ri;
    acc[0] += ri * ri;
  }
  if (reduce_last<1>(acc, cd.partial, cd.ticket, nb)) {
    sc->rnorm = sqrt(acc[0]);
    sc->cycle += 1;
  }
}

// ---- the Newton update -------------------------------------------------------------

// omega = min(1, fraction / max relative change of rho, p, nu_hat)  (implicit.py:54-81)
__global__ void __launch_bounds__(RED_THREADS) k_relax(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  const Canvas& c = cd.c;
  const Config& cfg = cd.cfg;
  const int N = c.ncanvas(), nv = c.nvar;
  int nb, lo, hi;
  if (!chunk_owner(N, nb, lo, hi)) return;
  const double g = cd.P.gamma;
  const double* __restrict__ U = cd.U;
  const double* __restrict__ dU = cd.x;
  double worst[1] = {0.0};
  if (cfg.max_relative_update > 0.0) {
    for (int idx = lo + threadIdx.x; idx < hi; idx += blockDim.x) {
      double rho = U[idx], u = U[N + idx] / rho, v = U[2 * N + idx] / rho;
      double p = (g - 1.0) * (U[3 * N + idx] - 0.5 * rho * (u * u + v * v));
      double de = dU[3 * N + idx] - u * dU[N + idx] - v * dU[2 * N + idx];
      double dp = (g - 1.0) * (de + 0.5 * (u * u + v * v) * dU[idx]);
      double w = nmax(fabs(dU[idx]) / rho, fabs(dp) / p);
      if (nv > 4) {
        double nh = U[4 * N + idx] / rho;
        double dnh = (dU[4 * N + idx] - nh * dU[idx]) / rho;
        w = nmax(w, fabs(dnh) / fmax(fabs(nh), 1.0));
      }
      worst[0] = nmax(worst[0], w);
    }
  }
  if (reduce_last<1, true>(worst, cd.partial, cd.ticket, nb)) {
    Scalars* sc = cd.sc;
    sc->worst = worst[0];
    if (cfg.max_relative_update > 0.0) {
      double q = cfg.max_relative_update / (worst[0] != worst[0] ? NAN : fmax(worst[0], 1e-300));
      sc->omega = q != q ? NAN : fmin(1.0, q);
    } else {
      sc->omega = 1.0;
    }
  }
}

// the linear reduction, physicality of the candidate, accept, the SER CFL ramp
__global__ void __launch_bounds__(RED_THREADS) k_accept(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  const Canvas& c = cd.c;
  const Config& cfg = cd.cfg;
  Scalars* sc = cd.sc;
  const int N = c.ncanvas(), nv = c.nvar, n = nv * N;
  int nb, lo, hi;
  if (!chunk_owner(n, nb, lo, hi)) return;
  const double g = cd.P.gamma, om = sc->omega;
  const double* __restrict__ U = cd.U;
  const double* __restrict__ dU = cd.x;
  const double* __restrict__ action = cd.action;
  const double* __restrict__ R = cd.R;
  double acc[3] = {0.0, 0.0, 0.0};  // |omega action + R|^2, |R|^2, bad cells
  for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    double t = om * action[i] + R[i];
    acc[0] += t * t;
    acc[1] += R[i] * R[i];
    if (!isfinite(om * dU[i])) acc[2] += 1.0;
    if (i < N) {
      double rho = U[i] + om * dU[i];
      double mx = U[N + i] + om * dU[N + i], my = U[2 * N + i] + om * dU[2 * N + i];
      double E = U[3 * N + i] + om * dU[3 * N + i];
      double u = mx / rho, v = my / rho;
      double p = (g - 1.0) * (E - 0.5 * rho * (u * u + v * v));
      bool ok = rho > 1e-10 && p > 1e-10 && isfinite(rho) && isfinite(p);
      if (!ok) acc[2] += 1.0;
    }
  }
  if (reduce_last<3>(acc, cd.partial, cd.ticket, nb)) {
    double lin = sqrt(acc[0]) / fmax(sqrt(acc[1]), 1e-300);
    bool physical = acc[2] == 0.0;
    bool accept = physical && lin < 1.0;
    double reduction = sc->res_prev / fmax(sc->norm, 1e-300);
    double cfl = sc->cfl, next;
    if (accept && lin < cfg.krylov_success && om >= 1.0)
      next = cfl * fmin(fmax(reduction, 1.0), cfg.cfl_growth);
    else if (accept)
      next = cfl;
    else
      next = cfl / cfg.cfl_cutback;
    sc->lin_red = lin;
    sc->accept = accept ? 1 : 0;
    sc->cfl = fmin(fmax(next, cfg.cfl_min), cfg.cfl_max);
    if (accept) sc->res_prev = sc->norm;
    sc->steps += 1;
    if (!accept) {
      sc->rejected += 1;
      sc->status |= ST_REJECTED;
    }
    if (!physical) sc->status |= ST_NONFINITE;
  }
}

__global__ void k_update(const CaseDev* __restrict__ cases) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled) return;
  const Scalars* sc = cd.sc;
  if (sc->accept == 0) return;
  const double om = sc->omega;
  double* __restrict__ U = cd.U;
  const double* __restrict__ dU = cd.x;
  const int n = cd.n_vec;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) U[i] = U[i] + om * dU[i];
}

// z = scale * src, optionally V_j = z rounded to the basis type: the Arnoldi step
// without a preconditioner (scale_on: by 1/|w| of the case)
template <class TV>
__global__ void k_scale_copy(const CaseDev* __restrict__ cases, int src_id, int scale_on, int vout_j, int out_id,
                             int check_active) {
  const CaseDev& cd = cases[blockIdx.y];
  if (!cd.enabled || (check_active && cd.sc->active == 0)) return;
  const int n = cd.n_vec;
  const double* __restrict__ src = buf(cd, src_id);
  double* __restrict__ z = buf(cd, out_id);
  TV* vout = vout_j >= 0 ? (TV*)cd.V + (size_t)vout_j * n : nullptr;
  const double s = scale_on ? cd.sc->inv_nrm : 1.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double x = s * src[i];
    if (vout != nullptr) {
      TV xv = TV(x);
      vout[i] = xv;
      x = double(xv);
    }
    z[i] = x;
  }
}

// ---- launch wrappers ------------------------------------------------------------------

// blocks of the basis passes of a case of n elements (and the largest block count any
// reduction uses: the size of a case's partial array)
int reduce_blocks(int n) { return max(max(2 * 148, chunk_blocks(n)), cgs_blocks(n)); }

static dim3 chunk_grid(const BatchDims& d) { return dim3(chunk_blocks(d.n_vec), d.n_cases); }
static dim3 stride_grid(const BatchDims& d) { return dim3(min((d.n_vec + 255) / 256, 148 * 4), d.n_cases); }

void launch_gmres_init(const CaseDev* cases, const BatchDims& d, cudaStream_t st) {
  k_gmres_init<<<chunk_grid(d), RED_THREADS, 0, st>>>(cases, d.n_slots);
}

void launch_cycle_start(const CaseDev* cases, const BatchDims& d, cudaStream_t st) {
  k_cycle_start<<<dim3(1, d.n_cases), 128, 0, st>>>(cases);
}

void launch_cycle_gate(const CaseDev* cases, const BatchDims& d, cudaGraphConditionalHandle gate,
                       unsigned long long* cycles, cudaStream_t st) {
  k_cycle_gate<<<1, 256, 0, st>>>(cases, d.n_cases, gate, cycles);
}

// The dense form where the launch has more blocks than SMs and they are short: at most 768
// elements for each block an SM is given, and 2560.  The three passes, registers and dense: two
// 385 x 97 SA cases (1311 elements a block) over 30 vectors 70 and 64 us, eight over 8, 15 and 30
// vectors 111 and 86, 191 and 151, 301 and 275 us; two 257 x 65 Euler cases (478) over 10 vectors 31 and 28 us,
// 32 of them 317 and 198 us; four 513 x 129 SA cases (2300) over 10 and 30 vectors 122 and 84, 239 and 232 us,
// but two over 30 vectors 125 and 144 us; four 769 x 193 cases (5110) over 30 vectors 448 and 500 us,
// eight 385 x 97 cases with one of those 410 and 516 us.  A case alone has at most a block an SM.
constexpr int ORTH_DENSE_EACH = 768, ORTH_DENSE_LONGEST = 2560;
static bool orth_dense(const BatchDims& d) {
  return d.orth_total > 148 && d.orth_chunk <= ORTH_DENSE_LONGEST &&
         148LL * d.orth_chunk <= (long long)ORTH_DENSE_EACH * d.orth_total;
}

template <int NK, int E, bool UPDATE>
static void orth_dots(const CaseDev* cases, const BatchDims& d, int k0, int count, int second, cudaStream_t st) {
  const dim3 grid(orth_blocks(d.n_vec), d.n_cases);
  if (orth_dense(d))
    k_orth_dots_dense<NK, UPDATE><<<grid, ORTH_THREADS, d.orth_chunk * sizeof(double), st>>>(cases, k0, count, second);
  else
    k_orth_dots<NK, E, UPDATE><<<grid, ORTH_THREADS, 0, st>>>(cases, k0, count, second);
}

static void orth_fp64(const CaseDev* cases, const BatchDims& d, int j, cudaStream_t st) {
  const int nk = j + 1;
  const dim3 grid(orth_blocks(d.n_vec), d.n_cases);
  auto dots = [&](int k0, int count, int second) {
    if (count <= 8) orth_dots<8, 4, false>(cases, d, k0, count, second, st);
    else if (count <= 16) orth_dots<16, 2, false>(cases, d, k0, count, second, st);
    else orth_dots<32, 1, false>(cases, d, k0, count, second, st);
  };
  auto update = [&](int first, int column) {
    if (orth_dense(d)) k_orth_update<true><<<grid, ORTH_THREADS, 0, st>>>(cases, nk, j, first, column);
    else k_orth_update<false><<<grid, ORTH_THREADS, 0, st>>>(cases, nk, j, first, column);
  };
  for (int k0 = 0; k0 < nk; k0 += ORTH_NK) dots(k0, min(ORTH_NK, nk - k0), 0);
  if (nk <= 8) {
    orth_dots<8, 4, true>(cases, d, 0, nk, 1, st);
  } else if (nk <= 16) {
    orth_dots<16, 2, true>(cases, d, 0, nk, 1, st);
  } else if (nk <= ORTH_NK) {
    orth_dots<32, 1, true>(cases, d, 0, nk, 1, st);
  } else {   // more vectors than a thread holds: the update, then the dots in slices
    update(1, 0);
    for (int k0 = 0; k0 < nk; k0 += ORTH_NK) dots(k0, min(ORTH_NK, nk - k0), 1);
  }
  update(0, 1);
}

template <int NK> static void mdot_fp32(const CaseDev* cases, const BatchDims& d, int j, cudaStream_t st) {
  const dim3 grid(d.cgs_blocks, d.n_cases);
  k_mdot_fp32<NK, 0><<<grid, RED_THREADS, 0, st>>>(cases, j + 1, j);
  k_mdot_fp32<NK, 1><<<grid, RED_THREADS, 0, st>>>(cases, j + 1, j);
  k_mdot_fp32<NK, 2><<<grid, RED_THREADS, 0, st>>>(cases, j + 1, j);
}

static void orth_fp32(const CaseDev* cases, const BatchDims& d, int j, cudaStream_t st) {
  const int nk = j + 1;
  if (nk <= 8) mdot_fp32<8>(cases, d, j, st);
  else if (nk <= 16) mdot_fp32<16>(cases, d, j, st);
  else if (nk <= 32) mdot_fp32<32>(cases, d, j, st);
  else mdot_fp32<64>(cases, d, j, st);
}

// orthogonalise w against V_0..V_j (CGS2) and append column j of H
void launch_arnoldi_orth(const CaseDev* cases, const BatchDims& d, bool fp32, int j, cudaStream_t st) {
  if (fp32) orth_fp32(cases, d, j, st);
  else orth_fp64(cases, d, j, st);
}

void launch_lstsq(const CaseDev* cases, const BatchDims& d, cudaStream_t st) {
  k_lstsq<<<dim3(1, d.n_cases), 32, 0, st>>>(cases);
}

void launch_combine(const CaseDev* cases, const BatchDims& d, bool fp32, cudaStream_t st) {
  if (fp32) k_combine<float><<<stride_grid(d), 256, 0, st>>>(cases);
  else k_combine<double><<<stride_grid(d), 256, 0, st>>>(cases);
}

void launch_cycle_end(const CaseDev* cases, const BatchDims& d, cudaStream_t st) {
  k_cycle_end<<<chunk_grid(d), RED_THREADS, 0, st>>>(cases);
}

void launch_scale_copy(const CaseDev* cases, const BatchDims& d, bool fp32, int src_id, int scale_on, int vout_j,
                       int out_id, int check_active, cudaStream_t st) {
  if (fp32 && vout_j >= 0)
    k_scale_copy<float><<<stride_grid(d), 256, 0, st>>>(cases, src_id, scale_on, vout_j, out_id, check_active);
  else
    k_scale_copy<double><<<stride_grid(d), 256, 0, st>>>(cases, src_id, scale_on, vout_j, out_id, check_active);
}

void launch_newton_update(const CaseDev* cases, const BatchDims& d, cudaStream_t st) {
  k_relax<<<dim3(chunk_blocks(d.cells), d.n_cases), RED_THREADS, 0, st>>>(cases);
  k_accept<<<chunk_grid(d), RED_THREADS, 0, st>>>(cases);
  k_update<<<stride_grid(d), 256, 0, st>>>(cases);
}

}  // namespace jr
