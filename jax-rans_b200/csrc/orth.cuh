// The sums of the orthogonalisation passes, 2D and 3D: many dot products at a time, a thread's
// own in registers, over the warp, the block and the blocks, in an order fixed by the sizes.
#pragma once
#include <cuda_runtime.h>

namespace jr {

// One block an SM: its threads' registers hold the basis entries in flight.
constexpr int ORTH_THREADS = 256, ORTH_BLOCKS = 148, ORTH_NK = 32;
// The elements a warp takes at a time where a warp takes a vector
constexpr int ORTH_ROUND = 2 * ORTH_THREADS;

// The NK sums of every lane over the warp, by a butterfly that halves the sums a lane holds at
// each exchange: afterwards lane l holds sum l * NK / 32 (NK < 32: every 32 / NK-th lane's) in
// acc[0].
template <int NK>
__device__ __forceinline__ void lane_sums(double (&acc)[NK], int lane) {
  int held = NK;
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    if (held >= 2) {
      const int half = held / 2;
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int k = 0; k < NK / 2; ++k)
        if (k < half) {
          const double send = upper ? acc[k] : acc[k + half], keep = upper ? acc[k + half] : acc[k];
          acc[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      held = half;
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    }
  }
}

// The sums of the nb blocks (blockIdx.x, ORTH_THREADS each; a block's in partial[b * NK + k], stored
// by any of its threads) in order, by the last block to finish; true there, with the totals in
// total[NK]
template <int NK>
__device__ bool finish_blocks(const double* partial, unsigned* ticket, int nb, double* total) {
  __shared__ double groups[ORTH_THREADS];
  __shared__ bool last;
  const int t = threadIdx.x;
  __threadfence();
  __syncthreads();
  if (t == 0) last = atomicAdd(ticket, 1u) == (unsigned)nb - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  constexpr int G = ORTH_THREADS / NK;
  const int k = t % NK, g = t / NK;
  double s = 0.0;
  for (int b = g; b < nb; b += 8 * G) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = b + u * G < nb ? __ldcg(partial + (size_t)(b + u * G) * NK + k) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += x[u];
  }
  groups[t] = s;
  __syncthreads();
  if (t < NK) {
    double v = groups[t];
    for (int q = 1; q < G; ++q) v += groups[q * NK + t];
    total[t] = v;
  }
  if (t == 0) *ticket = 0u;
  __syncthreads();
  return true;
}

// The same of sums[NK] of every thread: over the warp, then the block's warps in order, then the
// blocks
template <int NK>
__device__ bool finish_sums(double (&sums)[NK], double* partial, unsigned* ticket, int nb, double* total) {
  __shared__ double warps[ORTH_THREADS / 32][NK];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  lane_sums<NK>(sums, lane);
  if (lane % (32 / NK) == 0) warps[warp][lane / (32 / NK)] = sums[0];
  __syncthreads();
  if (t < NK) {
    double s = warps[0][t];
    for (int w = 1; w < ORTH_THREADS / 32; ++w) s += warps[w][t];
    partial[(size_t)blockIdx.x * NK + t] = s;
  }
  return finish_blocks<NK>(partial, ticket, nb, total);
}

}  // namespace jr
