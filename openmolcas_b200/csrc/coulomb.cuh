// The Coulomb half of the J/K build over one block of Cholesky vectors, FP64,
// for up to kJkMaxDens densities at once (used by the mixed and FP64 paths):
//   V[d nb + J] += sum_t L[t, J] dw_d[t]      (k_vmulti)
//   jrs_d[t]    += sum_J L[t, J] V[d nb + J]  (k_jacc_multi)
// Both read each vector element once for all densities; HBM bandwidth is the
// bound as soon as a block is larger than L2.
#pragma once
#include <cuda_runtime.h>

#include "mg_internal.h"

namespace mg {

constexpr int kJkMaxDens = 8;
constexpr int kVRows = 2048;  // vector elements per CTA of k_vmulti
constexpr int kVVecs = 4;     // vectors per CTA

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One CTA per (2048 rows, 4 vectors): every density value is loaded once for
// the four vectors and the grid covers the chip also for a block of 64 vectors.
// (One CTA per vector, its predecessor, left half of the SMs idle and each of
// the others with a single stream of loads: 193 us per block of 64 vectors at
// 403 functions with one further density; 8 us this way.)  The partial sums
// meet in V by atomics; the caller clears V.
template <int KD>
__global__ void __launch_bounds__(256) k_vmulti(const double* __restrict__ L, int64_t nrs, int nv, int nb,
                                                const double* __restrict__ dws, double* __restrict__ V) {
  __shared__ double red[kVVecs * KD][8];
  const int J0 = blockIdx.y * kVVecs;
  const int64_t t0 = (int64_t)blockIdx.x * kVRows + threadIdx.x;
  double acc[kVVecs][KD];
#pragma unroll
  for (int v = 0; v < kVVecs; ++v)
#pragma unroll
    for (int d = 0; d < KD; ++d) acc[v][d] = 0.0;
#pragma unroll 2
  for (int i = 0; i < kVRows / 256; ++i) {
    const int64_t t = t0 + 256 * i;
    if (t >= nrs) break;
    double x[kVVecs];
#pragma unroll
    for (int v = 0; v < kVVecs; ++v) x[v] = J0 + v < nv ? __ldg(L + t + nrs * (J0 + v)) : 0.0;
#pragma unroll
    for (int d = 0; d < KD; ++d) {
      const double w = __ldg(dws + (size_t)d * nrs + t);
#pragma unroll
      for (int v = 0; v < kVVecs; ++v) acc[v][d] = fma(x[v], w, acc[v][d]);
    }
  }
#pragma unroll
  for (int v = 0; v < kVVecs; ++v)
#pragma unroll
    for (int d = 0; d < KD; ++d) {
      const double s = warp_sum(acc[v][d]);
      if ((threadIdx.x & 31) == 0) red[v * KD + d][threadIdx.x >> 5] = s;
    }
  __syncthreads();
  if ((int)threadIdx.x < kVVecs * KD) {
    const int v = threadIdx.x / KD, d = threadIdx.x - v * KD;
    if (J0 + v < nv) {
      double s = 0.0;
      for (int w = 0; w < 8; ++w) s += red[threadIdx.x][w];
      atomicAdd(V + (size_t)d * nb + J0 + v, s);
    }
  }
}

// V += L^T dw for kd (1..8) packed densities dws (stride nrs), V at stride nb
static inline void launch_vmulti(const double* L, int64_t nrs, int nv, int nb, int kd, const double* dws, double* V,
                                 cudaStream_t st) {
  const dim3 grid((unsigned)((nrs + kVRows - 1) / kVRows), (nv + kVVecs - 1) / kVVecs);
  switch (kd) {
    case 1: k_vmulti<1><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 2: k_vmulti<2><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 3: k_vmulti<3><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 4: k_vmulti<4><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 5: k_vmulti<5><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 6: k_vmulti<6><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 7: k_vmulti<7><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
    case 8: k_vmulti<8><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, V); break;
  }
}

}  // namespace mg
