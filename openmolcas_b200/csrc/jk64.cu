// FP64 J/K from Cholesky vectors (CHO_LK_SCF, fock_util/cho_lk_scf.F90:14),
// the "plain FP64" path: all products in FP64 on the FP64 tensor pipe
// (mma.sync m8n8k4, the only FP64 matrix instruction of sm_100a).
//
// Per block of nb vectors and density:
//   k_half64   X_J = L_J C, one CTA per (64 rows, BN columns, vector); the
//              tiles of L_J are gathered from the rs-packed vector through the
//              inverse rs table, so no unpacked squares exist in memory
//   k_vmulti, k_jacc_multi (coulomb.cuh)   J
//   k_syrk64   K += X X^T over the lower tiles, the K extent split over the
//              CTAs so that a small matrix still fills the chip; every split
//              keeps its own partial tiles, summed in order by k_finish_k
// All sums run in a fixed order: a call gives the same bits every time (unless
// memory is short: blocks and splits then shrink, which changes the order).
// Measured, 300 functions, 1400 vectors, rank 41 (cuBLAS over blocks of 32
// unpacked squares before): half-transform 0.50 ms, 21 TFLOP/s (1.12 ms and 0.38
// ms of unpacking); exchange product 0.25 ms, 21 TFLOP/s (1.26 ms); whole Fock
// update 4.55 -> 1.18 ms with the parallel in-core decomposition.  1250 functions,
// 3789 vectors, rank 167: 146.8 -> 108.8 ms (27 TFLOP/s; the FP64 pipe peaks at
// 37).  Eight densities of rank 50 to 300 at 1820 functions, 699 vectors: 350 ms,
// against 336 with cuBLAS, where one unpacking served all eight.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "coulomb.cuh"
#include "kern_common.cuh"
#include "mg_internal.h"

namespace mg {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

constexpr int kKc = 16;  // K extent of a shared-memory chunk

// X_J = L_J C, a tile of 64 rows x 8 NT columns: 4 warps of 16 rows.  The rs
// indices are fetched two chunks and the vector elements one chunk ahead (two
// dependent loads per element).  Rows n..xld of X come out as zeros.
// Bound: the FP64 tensor pipe (82 percent busy at 896 functions, rank 320) and,
// close behind, the shared-memory and L1 pipe (per chunk of 16 k and 64 columns 1024
// clocks of products; some 900 of fragment reads, stores and gathers).  Hence the
// layout: A and B tiles have rows of 4 mod 16 doubles per k, so that the 16 lanes of
// a half-warp (4 k x 4 rows or columns) read 16 banks, and B's rows are shifted by
// one double after every fourth, so that a store (16 k of one column) has 16, too
// (it had 4: 1820 functions, 699 vectors, rank 300, 54.2 -> 52.1 ms).  The last
// column tile forms only the eights of columns there are (52.1 -> 48.1 ms; rank 193
// 37.0 -> 32.8).  Two such groups of warps over 112 columns, which halve the gathers
// per product, were no faster: 48.9 ms, rank 229 40.9 against 37.0.
template <int NT>
__global__ void __launch_bounds__(128) k_half64(const double* __restrict__ L, int64_t nrs,
                                                   const int* __restrict__ inv, int n, const double* __restrict__ C,
                                                   int r, double* __restrict__ X, int xld) {
  constexpr int BN = 8 * NT, SA = 68, SB = BN % 16 ? BN + 12 : BN + 4, SB4 = 4 * SB + 1;
  __shared__ double As[2][kKc][SA];
  __shared__ double Bs[2][kKc / 4 * SB4];
  const int a0 = blockIdx.x * 64, c0 = blockIdx.y * BN, J = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nj = min(NT, (r - c0 + 7) >> 3);  // eights of columns
  const double* LJ = L + nrs * J;
  const int row = tid & 63, kr = tid >> 6;  // A: row, k = kr + 2 i
  const int bk = tid & 15, bc = tid >> 4;   // B: k, column bc + 8 i
  const int bo = (bk >> 2) * SB4 + (bk & 3) * SB + bc;
  const int nch = (n + kKc - 1) / kKc;
  int idx[8];
  double av[8], bv[NT];
  auto load_idx = [&](int ch) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int b = ch * kKc + kr + 2 * i;
      idx[i] = (a0 + row < n && b < n) ? __ldg(inv + (size_t)b * n + a0 + row) : -1;
    }
  };
  auto load_val = [&](int ch) {
#pragma unroll
    for (int i = 0; i < 8; ++i) av[i] = idx[i] >= 0 ? __ldg(LJ + idx[i]) : 0.0;
    const int b = ch * kKc + bk;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const int c = c0 + bc + 8 * i;
      bv[i] = (b < n && c < r) ? __ldg(C + (size_t)c * n + b) : 0.0;
    }
  };
  double acc[2][NT][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  auto product = [&](int s, auto cols) {
    constexpr int N = decltype(cols)::value;
    if constexpr (N <= NT) {
#pragma unroll
      for (int ks = 0; ks < kKc / 4; ++ks) {
        const double* ap = &As[s][4 * ks + (lane & 3)][warp * 16 + (lane >> 2)];
        const double* bp = &Bs[s][ks * SB4 + (lane & 3) * SB + (lane >> 2)];
        const double f0 = ap[0], f1 = ap[8];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const double b = bp[8 * j];
          dmma(acc[0][j], f0, b);
          dmma(acc[1][j], f1, b);
        }
      }
    }
  };
  load_idx(0);
  load_val(0);
  load_idx(1);
  for (int ch = 0; ch < nch; ++ch) {
    const int s = ch & 1;
#pragma unroll
    for (int i = 0; i < 8; ++i) As[s][kr + 2 * i][row] = av[i];
#pragma unroll
    for (int i = 0; i < NT; ++i) Bs[s][bo + 8 * i] = bv[i];
    __syncthreads();
    if (ch + 1 < nch) {
      load_val(ch + 1);
      load_idx(ch + 2);
    }
    switch (nj) {  // (unrolled for every width: a test per eight columns costs a tenth)
      case 1: product(s, std::integral_constant<int, 1>{}); break;
      case 2: product(s, std::integral_constant<int, 2>{}); break;
      case 3: product(s, std::integral_constant<int, 3>{}); break;
      case 4: product(s, std::integral_constant<int, 4>{}); break;
      case 5: product(s, std::integral_constant<int, 5>{}); break;
      case 6: product(s, std::integral_constant<int, 6>{}); break;
      case 7: product(s, std::integral_constant<int, 7>{}); break;
      case 8: product(s, std::integral_constant<int, 8>{}); break;
    }
  }
#pragma unroll
  for (int j = 0; j < NT; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = c0 + 8 * j + 2 * (lane & 3) + e;
      if (j < nj && c < r) {
        double* x = X + ((size_t)J * r + c) * xld + a0 + warp * 16 + (lane >> 2);
        x[0] = acc[0][j][e];
        x[8] = acc[1][j][e];
      }
    }
}

__device__ __forceinline__ void cp16(void* dst, const void* src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int sz = valid ? 16 : 0;  // 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(sz) : "memory");
}

// P[split][tile] (+)= X X^T (lower tiles of 64 x 64, column-major): X
// column-major with leading dimension xld (a multiple of 64; rows n.. zero), kt
// columns.  blockIdx.x: lower tile, blockIdx.y: split, a range of cps chunks of
// 16 columns.  Three-stage cp.async ring; 2 x 2 warps of 32 x 32.  first: write
// instead of add.  Tiles of 128 in eight warps halve the L2 reads but were slower
// at every size tried (whole J/K call, ms): 644 functions 1.40 against 1.25, 896
// 4.04 against 3.83, 1246 16.1 against 15.8, 2100 123 against 109.
constexpr int kSyTile = 64;

__global__ void __launch_bounds__(128) k_syrk64(const double* __restrict__ X, int xld, int64_t kt, int cps, int first,
                                                double* __restrict__ P) {
  constexpr int BT = kSyTile, NWM = 2, FM = 4, FN = 4, T = 128, ST = BT + 4, NSTG = 3;
  extern __shared__ __align__(16) double sy_smem[];
  int ti = (int)((sqrtf(8.0f * blockIdx.x + 1.0f) - 1.0f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
  while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
  const int tj = (int)blockIdx.x - ti * (ti + 1) / 2;
  const bool diag = ti == tj;
  const int64_t nch_all = (kt + kKc - 1) / kKc;
  const int64_t ch0 = (int64_t)blockIdx.y * cps;
  const int nch = (int)min((int64_t)cps, nch_all - ch0);
  if (nch <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp % NWM, wn = warp / NWM;
  auto stage = [&](int s, int op) { return sy_smem + (size_t)(2 * s + op) * kKc * ST; };
  auto load = [&](int ch, int s) {
    const int64_t k0 = (ch0 + ch) * kKc;
#pragma unroll
    for (int i = tid; i < kKc * BT / 2; i += T) {
      const int kk = i / (BT / 2), a = 2 * (i % (BT / 2));
      const bool ok = k0 + kk < kt;
      const double* src = X + (size_t)(ok ? k0 + kk : 0) * xld + a;
      cp16(stage(s, 0) + kk * ST + a, src + ti * BT, ok);
      if (!diag) cp16(stage(s, 1) + kk * ST + a, src + tj * BT, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[FM][FN][2];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  load(0, 0);
  if (nch > 1) load(1, 1);
  else asm volatile("cp.async.commit_group;" ::: "memory");
  for (int ch = 0; ch < nch; ++ch) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (ch + 2 < nch) load(ch + 2, (ch + 2) % NSTG);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const double* A = stage(ch % NSTG, 0);
    const double* B = diag ? A : stage(ch % NSTG, 1);
#pragma unroll
    for (int ks = 0; ks < kKc / 4; ++ks) {
      const double* ap = A + (4 * ks + (lane & 3)) * ST + wm * FM * 8 + (lane >> 2);
      const double* bp = B + (4 * ks + (lane & 3)) * ST + wn * FN * 8 + (lane >> 2);
      double fa[FM];
#pragma unroll
      for (int i = 0; i < FM; ++i) fa[i] = ap[8 * i];
#pragma unroll
      for (int j = 0; j < FN; ++j) {
        const double fb = bp[8 * j];
#pragma unroll
        for (int i = 0; i < FM; ++i) dmma(acc[i][j], fa[i], fb);
      }
    }
  }
  double* Pt = P + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * BT * BT;
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        double* p = Pt + (size_t)((wn * FN + j) * 8 + 2 * (lane & 3) + e) * BT + (wm * FM + i) * 8 + (lane >> 2);
        *p = first ? acc[i][j][e] : *p + acc[i][j][e];
      }
}

// K (both triangles) from the splits' partial lower tiles, in order
__global__ void k_finish_k(const double* __restrict__ P, int bt, int ntile, int nsplit, int n, double* __restrict__ K) {
  const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (o >= (int64_t)n * n) return;
  const int a = (int)(o % n), b = (int)(o / n);
  if (a < b) return;
  const int ti = a / bt, tj = b / bt;
  const double* p = P + (size_t)(ti * (ti + 1) / 2 + tj) * bt * bt + (size_t)(b % bt) * bt + a % bt;
  double s = 0.0;
  for (int q = 0; q < nsplit; ++q) s += p[(size_t)q * ntile * bt * bt];
  K[(size_t)b * n + a] = s;
  K[(size_t)a * n + b] = s;
}

static int launch_half64(int nt, dim3 grid, const double* L, int64_t nrs, const int* inv, int n, const double* C,
                         int r, double* X, int xld, cudaStream_t st) {
  switch (nt) {
    case 1: k_half64<1><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 2: k_half64<2><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 3: k_half64<3><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 4: k_half64<4><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 5: k_half64<5><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 6: k_half64<6><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 7: k_half64<7><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    case 8: k_half64<8><<<grid, 128, 0, st>>>(L, nrs, inv, n, C, r, X, xld); break;
    default: return MG_ERR_ARG;
  }
  return 0;
}

constexpr int kSyrkSmem = 3 * 2 * kKc * (kSyTile + 4) * 8;

int jk_fp64(Handle* h, const double* d_C, int r, double* d_J, double* d_K, cudaStream_t st) {
  return jk_fp64_batch(h, 1, &d_C, &r, &d_J, &d_K, st);
}

int jk_fp64_batch(Handle* h, int k, const double* const* Cs, const int* rs_, double* const* Js, double* const* Ks,
                  cudaStream_t st) {
  ChoState* c = h->cho;
  const int64_t nrs = cho_nrs(c);
  const int M = cho_nvec(c), n = h->nbf;
  if (k < 1 || k > kJkMaxDens) { h->err = "FP64 J/K: 1..8 densities per batch"; return MG_ERR_ARG; }
  int rmax = 0;
  for (int d = 0; d < k; ++d) {
    if (!Cs[d] || !Js[d] || !Ks[d] || rs_[d] < 1) { h->err = "FP64 J/K: a density of the batch has no factor or outputs"; return MG_ERR_ARG; }
    rmax = std::max(rmax, rs_[d]);
  }
  if (M == 0) return jk_no_vectors(h, k, Js, Ks, st);
  const int* inv = cho_inv_dev(c);
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
  constexpr int bt = kSyTile;
  const int xld = (n + bt - 1) / bt * bt;
  // vectors per block: a power of two (storage blocks of 1024 are not
  // straddled) that keeps X at or below 256 MB, at least 16
  int nb = 1024;
  while (nb > 16 && (size_t)nb * rmax * xld * 8 > ((size_t)256 << 20)) nb /= 2;
  nb = std::min(nb, cho_vec_block());
  const int nt = xld / bt, ntile = nt * (nt + 1) / 2, nr = vmulti_ranges(nrs);
  int nbm = 0;                       // vectors X holds
  int per_sm = 8;                    // CTAs per SM that the K splits aim at
  // K splits of a full block of rank r, at least 8 chunks each: of that number and
  // up to twice as many, the first that fills the last wave of CTAs (four of 52 KB
  // are resident per SM) within 3 percent of the best (exchange product at 1246
  // functions, rank 300, 210 tiles: five splits 9.2 ms, eight 8.7)
  auto splits = [&](int r, int& cps) {
    const int64_t nch = ((int64_t)nbm * r + kKc - 1) / kKc;
    const int64_t want = std::max<int64_t>(1, (int64_t)nsm * per_sm / ntile);
    int64_t ns = std::max<int64_t>(1, std::min<int64_t>(want, nch / 8));
    const int64_t most = per_sm ? std::max<int64_t>(ns, std::min<int64_t>(2 * ns, nch / 8)) : ns;
    auto fill = [&](int64_t q) {
      const int64_t slots = 4 * (int64_t)nsm, ctas = q * ntile;
      return (double)ctas / (double)((ctas + slots - 1) / slots * slots);
    };
    double best = 0.0;
    for (int64_t q = ns; q <= most; ++q) best = std::max(best, fill(q));
    while (fill(ns) < best - 0.03) ++ns;
    cps = (int)((nch + ns - 1) / ns);
    return (int)((nch + cps - 1) / cps);
  };
  // Memory short: blocks of half as many vectors, down to 16, then half as many
  // splits, until the workspace can be had.
  int cps = 0, jsplit = 0;
  size_t nx = 0, np = 0, nj = 0, nvp = 0;
  double* ws = nullptr;
  for (;;) {
    nbm = std::min(nb, M);
    int smax = 1;
    for (int d = 0; d < k; ++d) smax = std::max(smax, splits(rs_[d], cps));
    jsplit = jacc_splits(nrs, nbm, nsm);
    nx = (size_t)nbm * rmax * xld;
    np = (size_t)smax * ntile * bt * bt;
    nj = (size_t)jsplit * k * nrs;
    nvp = (size_t)nr * k * nb;
    ws = (double*)ws_get(h, sizeof(double) * (nx + np + nj + nvp + (size_t)nb * k + (size_t)nrs * k), st);
    if (ws || (nb <= 16 && per_sm == 0)) break;
    if (nb > 16) nb /= 2;
    else per_sm /= 2;
  }
  if (!ws) { h->err = "jk workspace allocation failed"; return MG_ERR_MEMORY; }
  double* X = ws;  // first: 16-byte aligned columns for cp.async (xld even)
  double* P = X + nx;
  double* jrs = P + np;
  double* Vp = jrs + nj;
  double* V = Vp + nvp;
  double* dw = V + (size_t)nb * k;
  auto count = [](int m) { g_launches.fetch_add(m, std::memory_order_relaxed); };
  if (!smem_attr_once((const void*)k_syrk64, kSyrkSmem)) {
    h->err = "FP64 J/K: shared-memory limit could not be raised";
    return MG_ERR_CUDA;
  }
  // Coulomb: all densities in one pass over the vectors
  for (int d = 0; d < k; ++d)
    k_density_rs<<<nb256(nrs), 256, 0, st>>>(cho_rs_a_dev(c), cho_rs_b_dev(c), nrs, Cs[d], n, rs_[d],
                                             dw + (size_t)d * nrs);
  cudaMemsetAsync(jrs, 0, sizeof(double) * nj, st);
  count(k);
  for (int J0 = 0; J0 < M; J0 += nb) {
    const int nv = std::min(nb, M - J0);
    const double* Lb = cho_vec_ptr(c, J0, nv, st, h);
    if (!Lb) { h->err = "vector block straddles storage blocks"; return MG_ERR_ARG; }
    launch_vmulti(Lb, nrs, nv, nb, k, dw, Vp, V, st);
    launch_jacc(Lb, nrs, nv, nb, k, jsplit, V, jrs, st);
    count(3);
  }
  for (int d = 0; d < k; ++d)
    k_finish_j<<<nb256((int64_t)n * n), 256, 0, st>>>(inv, jrs + (size_t)d * nrs, jsplit, (int64_t)k * nrs, n, Js[d]);
  count(k);
  // exchange, one density after another
  for (int d = 0; d < k; ++d) {
    const int r = rs_[d], nsplit = splits(r, cps);
    const int nct = (r + 63) / 64, nt8 = ((r + nct - 1) / nct + 7) / 8;
    int used = 0;  // splits that hold something
    for (int J0 = 0; J0 < M; J0 += nb) {
      const int nv = std::min(nb, M - J0);
      const double* Lb = cho_vec_ptr(c, J0, nv, st, h);
      launch_half64(nt8, dim3(xld / 64, nct, nv), Lb, nrs, inv, n, Cs[d], r, X, xld, st);
      const int64_t kt = (int64_t)nv * r, nch = (kt + kKc - 1) / kKc;
      const dim3 grid(ntile, (unsigned)std::min<int64_t>(nsplit, (nch + cps - 1) / cps));
      k_syrk64<<<grid, 128, kSyrkSmem, st>>>(X, xld, kt, cps, J0 == 0, P);
      used = std::max(used, (int)grid.y);
      count(2);
    }
    k_finish_k<<<nb256((int64_t)n * n), 256, 0, st>>>(P, bt, ntile, used, n, Ks[d]);
    count(1);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : MG_ERR_CUDA;
}

}  // namespace mg
