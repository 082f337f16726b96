// The Coulomb half of the J/K build over one block of Cholesky vectors, FP64,
// for up to kJkMaxDens densities at once (used by the mixed and FP64 paths):
//   V[d nb + J] = sum_t L[t, J] dw_d[t]       (k_vmulti, k_vsum)
//   jrs_d[t]    += sum_J L[t, J] V[d nb + J]  (k_jacc_multi)
// Both read each vector element once for all densities; HBM bandwidth is the
// bound as soon as a block is larger than L2.  Also the packed density before
// and the dense J and K after.
#pragma once
#include <cuda_runtime.h>

#include "mg_internal.h"

namespace mg {

static inline unsigned nb256(int64_t n) { return (unsigned)((n + 255) / 256); }

// dw[t] = w_t sum_k C[a_t, k] C[b_t, k], w = 2 for a != b, 1 on the diagonal
// (the packed density D = C C^T; C column-major n x r)
static __global__ void k_density_rs(const int* __restrict__ rs_a, const int* __restrict__ rs_b, int64_t nrs,
                             const double* __restrict__ C, int n, int r, double* __restrict__ dw) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nrs) return;
  const int a = rs_a[t], b = rs_b[t];
  double s0 = 0.0, s1 = 0.0;
  int k = 0;
  for (; k + 2 <= r; k += 2) {
    const double* c = C + (size_t)k * n;
    s0 = fma(__ldg(c + a), __ldg(c + b), s0);
    s1 = fma(__ldg(c + n + a), __ldg(c + n + b), s1);
  }
  if (k < r) s0 = fma(__ldg(C + (size_t)k * n + a), __ldg(C + (size_t)k * n + b), s0);
  dw[t] = (a == b ? 1.0 : 2.0) * (s0 + s1);
}

// J from its rs-packed form (the splits' shares in order; zero where no rows are
// stored): jrs at stride js per split
static __global__ void k_finish_j(const int* __restrict__ inv, const double* __restrict__ jrs, int split, int64_t js,
                                  int n, double* __restrict__ J) {
  const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (o >= (int64_t)n * n) return;
  const int t = inv[o];
  double s = 0.0;
  if (t >= 0)
    for (int q = 0; q < split; ++q) s += jrs[q * js + t];
  J[o] = s;
}

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
// 403 functions with one further density; 8 us this way.  Eight vectors per CTA:
// 5.3 instead of 3.9 ms a call at 1250 functions, one density.)  The partial sums of
// the row ranges go to Vp[range][KD nb] and are added in order by k_vsum, so the
// result does not depend on the order in which the CTAs run.
template <int KD>
__global__ void __launch_bounds__(256) k_vmulti(const double* __restrict__ L, int64_t nrs, int nv, int nb,
                                                const double* __restrict__ dws, double* __restrict__ Vp) {
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
      Vp[(size_t)blockIdx.x * KD * nb + (size_t)d * nb + J0 + v] = s;
    }
  }
}

// V[o] = sum over the nr row ranges of Vp[range][o], one warp per o
static __global__ void k_vsum(const double* __restrict__ Vp, int nr, int nv, int nb, int kd, double* __restrict__ V) {
  const int o = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (o >= kd * nb || o % nb >= nv) return;
  double s = 0.0;
  for (int r = lane; r < nr; r += 32) s += Vp[(size_t)r * kd * nb + o];
  s = warp_sum(s);
  if (lane == 0) V[o] = s;
}

static inline int vmulti_ranges(int64_t nrs) { return (int)((nrs + kVRows - 1) / kVRows); }

// V = L^T dw for kd (1..8) packed densities dws (stride nrs), V at stride nb;
// Vp: vmulti_ranges(nrs) kd nb doubles of scratch
static inline void launch_vmulti(const double* L, int64_t nrs, int nv, int nb, int kd, const double* dws, double* Vp,
                                 double* V, cudaStream_t st) {
  const dim3 grid((unsigned)((nrs + kVRows - 1) / kVRows), (nv + kVVecs - 1) / kVVecs);
  switch (kd) {
    case 1: k_vmulti<1><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 2: k_vmulti<2><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 3: k_vmulti<3><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 4: k_vmulti<4><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 5: k_vmulti<5><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 6: k_vmulti<6><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 7: k_vmulti<7><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
    case 8: k_vmulti<8><<<grid, 256, 0, st>>>(L, nrs, nv, nb, dws, Vp); break;
  }
  k_vsum<<<(kd * nb + 7) / 8, 256, 0, st>>>(Vp, (int)grid.x, nv, nb, kd, V);
}

// One thread per row; the vectors are split over blockIdx.y (a small system has
// too few rows to fill the chip or to hide the latency of one serial pass), and
// every split adds into its own jrs, summed in order by the last kernel.
template <int KD>
__global__ void __launch_bounds__(256) k_jacc_multi(const double* __restrict__ L, int64_t nrs, int nv, int nb,
                                                    const double* __restrict__ V, double* __restrict__ jrs) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nrs) return;
  const int per = (nv + gridDim.y - 1) / gridDim.y;
  const int J0 = blockIdx.y * per, J1 = min(nv, J0 + per);
  double acc[KD];
#pragma unroll
  for (int d = 0; d < KD; ++d) acc[d] = 0.0;
#pragma unroll 8
  for (int J = J0; J < J1; ++J) {
    const double x = __ldg(L + t + nrs * J);
#pragma unroll
    for (int d = 0; d < KD; ++d) acc[d] = fma(x, __ldg(V + (size_t)d * nb + J), acc[d]);
  }
#pragma unroll
  for (int d = 0; d < KD; ++d) jrs[((size_t)blockIdx.y * KD + d) * nrs + t] += acc[d];
}

// splits of the vectors of a block of nb: eight CTAs per SM in all, at least 16
// vectors each
static inline int jacc_splits(int64_t nrs, int nb, int nsm) {
  const int64_t s = 8 * (int64_t)nsm / ((nrs + 255) / 256);
  return (int)(s < 1 || nb < 32 ? 1 : s > nb / 16 ? nb / 16 : s);
}

// jrs[split][k][nrs] += L V for k (1..8) densities
static inline void launch_jacc(const double* L, int64_t nrs, int nv, int nb, int k, int split, const double* V,
                               double* jrs, cudaStream_t st) {
  const dim3 grid((unsigned)((nrs + 255) / 256), split);
  switch (k) {
    case 1: k_jacc_multi<1><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 2: k_jacc_multi<2><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 3: k_jacc_multi<3><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 4: k_jacc_multi<4><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 5: k_jacc_multi<5><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 6: k_jacc_multi<6><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 7: k_jacc_multi<7><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
    case 8: k_jacc_multi<8><<<grid, 256, 0, st>>>(L, nrs, nv, nb, V, jrs); break;
  }
}

}  // namespace mg
