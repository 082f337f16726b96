// Coulomb / exchange matrices from Cholesky vectors (the CHO_LK_SCF build,
// fock_util/cho_lk_scf.F90:14) on the GPU.
//
//   D = C C^T (C: nbf x r, the Cholesky/orbital factor of the density, as
//   ChoSCF_Drv passes it, scf/choscf_drv.F90:115-116)
//   J_ab = sum_J L_ab,J V_J,  V_J = sum_cd L_cd,J D_cd     (cho_lk_scf.F90:442-449)
//   K_ab = sum_J sum_k X_J[a,k] X_J[b,k],  X_J = L_J C      (cho_lk_scf.F90:507-830)
//
// Mixed path: the FP64 vectors are cut into 8-bit slices per row (oz_gemm.cuh
// gives the scheme; s slices for the half-transform, sk for the exchange
// product, whose error dominates) and both exchange GEMMs run on the tcgen05
// tensor cores in 8-bit integers with exact INT32 accumulation: per block of
// vectors, a slicing kernel unpacks the rs-packed L_J into sliced dense
// squares, the
// half-transform X_J = L_J C writes X in FP64, X is sliced per row over the
// block, and the exchange product K += X X^T runs over groups of blocks
// (lower-triangle tiles, CTA-private FP64 tiles, FP64 atomics into K).  J
// is FP64 throughout.
//
// The FP64 path is in jk64.cu.
// LK screening is not applied (dense tensor work is cheaper on the GPU than
// the screening bookkeeping); the result equals the unscreened reference.
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "coulomb.cuh"
#include "kern_common.cuh"
#include "mg_internal.h"
#include "oz_gemm.cuh"

namespace mg {

__global__ void k_symmetrize_lower(double* __restrict__ K, int n) {
  int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (o >= (int64_t)n * n) return;
  const int i = (int)(o % n), j = (int)(o / n);
  if (i > j) K[(size_t)i * n + j] = K[(size_t)j * n + i];  // column-major lower -> full
}

// F += J - factxi K (CHO_LK_SCF's FLT update)
__global__ void k_fock_acc(double* __restrict__ F, const double* __restrict__ J, const double* __restrict__ K,
                           double factxi, int64_t n) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < n) F[t] += J[t] - factxi * K[t];
}

// J = K = 0 of a decomposition without vectors (the threshold above the largest
// diagonal: possibly without rows, too)
int jk_no_vectors(Handle* h, int k, double* const* Js, double* const* Ks, cudaStream_t st) {
  const size_t bytes = sizeof(double) * (size_t)h->nbf * h->nbf;
  for (int d = 0; d < k; ++d)
    if (cudaMemsetAsync(Js[d], 0, bytes, st) != cudaSuccess || cudaMemsetAsync(Ks[d], 0, bytes, st) != cudaSuccess) {
      h->err = std::string("J/K: clearing the outputs: ") + cudaGetErrorString(cudaGetLastError());
      return MG_ERR_CUDA;
    }
  return 0;
}

int fock_accumulate(double* F, const double* J, const double* K, double factxi, int64_t n, cudaStream_t st) {
  k_fock_acc<<<nb256(n), 256, 0, st>>>(F, J, K, factxi, n);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  if (cudaGetLastError() != cudaSuccess) return MG_ERR_CUDA;
  return cudaStreamSynchronize(st) == cudaSuccess ? 0 : MG_ERR_CUDA;
}

// ------------------------------------------------------------ mixed path
// Slicing of one value x of a row with exponent e (y = x 2^-e in (-1, 1))
// into S 8-bit pieces (oz_gemm.cuh): y as the S-byte two's-complement
// fixed-point integer Y = floor(y 2^(8S-1)), its lowest byte rounded to
// nearest where that does not carry out of the byte; slice p is byte S-1-p
// of Y (S_0 the signed top byte, U_p unsigned), so every slice but the last
// is the floor digit and the dropped tail is below one unit of the last.
struct OzScale {
  double lo, hi;  // 2^(8S-1-e) as two factors, each a normal double
};

template <int S>
__device__ __forceinline__ OzScale oz_scale(int e) {
  const int k = 8 * S - 1 - e, k1 = k >> 1;  // e in [-1073, 1024]: both halves in range
  return {oz_pow2(k1), oz_pow2(k - k1)};
}

template <int S>
__device__ __forceinline__ long long oz_fixed(double x, OzScale sc) {
  const double z = (x * sc.lo) * sc.hi;  // exact power-of-two scaling, |z| < 2^(8S-1)
  long long y;
  double frac;
  if (S <= 6) {
    // |z| < 2^47: adding 1.5 2^52 rounded down leaves floor(z) in the low
    // mantissa bits (the unit in the last place is 1 there), on the adder
    constexpr double kM = 6755399441055744.0;  // 1.5 2^52
    const double t = __dadd_rd(z, kM);
    y = (__double_as_longlong(t) & ((1ll << 52) - 1)) - (1ll << 51);
    frac = z - (t - kM);  // both differences exact
  } else {
    y = __double2ll_rd(z);
    frac = z - (double)y;  // exact: z is integral beyond 2^52
  }
  if (frac >= 0.5 && (y & 255) != 255) ++y;
  return y;
}

// slice p of 8 consecutive values: out[p] holds their bytes S-1-p
template <int S>
__device__ __forceinline__ void oz_pack8(const long long (&y)[8], uint2 (&out)[S]) {
#pragma unroll
  for (int p = 0; p < S; ++p) {
    const int sh = 8 * (S - 1 - p);
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      lo |= (uint32_t)((y[u] >> sh) & 255) << (8 * u);
      hi |= (uint32_t)((y[4 + u] >> sh) & 255) << (8 * u);
    }
    out[p] = make_uint2(lo, hi);
  }
}

// f(std::integral_constant<int, s>) for s = 2..kOzMaxSlices
template <typename F>
static bool oz_with_slices(int s, F&& f) {
  switch (s) {
    case 2: f(std::integral_constant<int, 2>{}); return true;
    case 3: f(std::integral_constant<int, 3>{}); return true;
    case 4: f(std::integral_constant<int, 4>{}); return true;
    case 5: f(std::integral_constant<int, 5>{}); return true;
    case 6: f(std::integral_constant<int, 6>{}); return true;
    case 7: f(std::integral_constant<int, 7>{}); return true;
    case 8: f(std::integral_constant<int, 8>{}); return true;
  }
  return false;
}
static_assert(kOzMaxSlices == 8, "oz_with_slices covers 2..8 slices");

__device__ __forceinline__ int oz_exponent(double m) {
  int e = 0;
  if (m > 0.0) frexp(m, &e);
  return e;
}

__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Row exponents of the square Cholesky vectors, computed once per
// decomposition: one warp per row (J, a) gathers L_J[a, 0..n) from the
// rs-packed FP64 vectors through the inverse rs table and stores the frexp
// exponent of its largest |element| (0 for a zero row and for a >= n).
__global__ void k_oz_lexp(const int* __restrict__ inv, int n, int64_t nrs, const double* __restrict__ L, int nb,
                          int ld, short* __restrict__ eL) {
  const int lane = threadIdx.x & 31;
  const int64_t row = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= (int64_t)nb * ld) return;
  const int J = (int)(row / ld), a = (int)(row - (int64_t)J * ld);
  const double* LJ = L + nrs * J;
  double m = 0.0;
  if (a < n)
    for (int b = lane; b < n; b += 32) {
      const int t = inv[(size_t)a * n + b];  // -1: not stored (zero)
      if (t >= 0) m = fmax(m, fabs(LJ[t]));
    }
  m = warp_max(m);
  if (lane == 0) eL[row] = (short)max(-32000, oz_exponent(m));
}

// L slicing: the squares of a block of rs-packed vectors, cut into slices.  One
// CTA per (128 AOs b, 32 AOs a, kOzVecs vectors), two threads per row b with 16
// columns a each.  The rs indices of a thread's 16 elements are looked up once
// for all its vectors (the inverse rs table), all 16 vector elements of a
// vector are in flight at once.  L_J is symmetric, so L_J[a, b] is row b,
// column a: 16 consecutive K bytes of row b of every slice, cut with row b's
// cached exponent and packed in registers; the two threads of a row write its
// 32 bytes of a slice, so a warp's store is 512 contiguous bytes (the blocked
// layout of oz_blk_off).  The grid covers the K steps that the half-transform
// reads: the padding a >= n of the last one is written as zeros, as are the rows
// b >= n.
// Cut: z = x 2^(8S-1-e), rounded to the nearest integer (at most half a unit of
// the last slice; 2^(8S-1) itself, from a value just below it, becomes the
// integer before).  For S <= 6 adding 1.5 2^52 leaves the two's-complement
// integer in the low mantissa bits: three FP64 operations per element.
// Bound: HBM, S bytes written per element of the squares and the packed vectors
// read; 1250 functions, 3789 vectors, S = 6: 10.1 ms a call, 54 GB (28.6 ms with a
// shell-pair lookup per element and vector, a floor, a rounding test and the
// Coulomb contraction in the same kernel).
constexpr int kOzCutRows = 128;  // AOs b per CTA
constexpr int kOzCutCols = 32;   // AOs a per CTA: one MMA K step
constexpr int kOzVecs = 4;       // vectors per CTA
// sliced squares of one launch at most
constexpr size_t kOzGroupBytes = (size_t)512 << 20;

template <int S>
__global__ void __launch_bounds__(2 * kOzCutRows) k_oz_slice_l(const int* __restrict__ inv, int n, int64_t nrs,
                                                               const double* __restrict__ L, int nv, int ld,
                                                               int64_t slice, const short* __restrict__ eL,
                                                               uint8_t* __restrict__ LS, int* __restrict__ eA) {
  const int b = blockIdx.x * kOzCutRows + (threadIdx.x >> 1);
  const int a0 = blockIdx.y * kOzCutCols + 16 * (threadIdx.x & 1);
  const int J0 = blockIdx.z * kOzVecs, J1 = min(nv, J0 + kOzVecs);
  int idx[16];
#pragma unroll
  for (int r = 0; r < 16; ++r) idx[r] = (b < n && a0 + r < n) ? __ldg(inv + (size_t)(a0 + r) * n + b) : -1;
  constexpr double kM = 6755399441055744.0;                  // 1.5 2^52
  constexpr double zmax = (double)((1ull << (8 * (S < 7 ? S : 6) - 1)) - 1);
  for (int J = J0; J < J1; ++J) {
    const double* LJ = L + nrs * J;
    const int64_t row = (int64_t)J * ld + b;
    const int e = eL[row];
    if (a0 == 0) eA[row] = e;
    double x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = idx[r] >= 0 ? __ldg(LJ + idx[r]) : 0.0;
    // 2^(8S-1-e): one normal factor except for rows below 2^-950
    const int k = 8 * S - 1 - e, k1 = min(k, 1000);
    const double f1 = oz_pow2(k1);
    if (k != k1) {
      const double f2 = oz_pow2(k - k1);
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r] *= f2;
    }
    uint32_t w[S][4];  // slice p, columns a0 + 4 g .. + 3 (one byte each)
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t lo[4], hi[4];  // the two words of the integers of four columns
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double z = x[4 * g + q] * f1;
        long long y;
        if (S <= 6) y = __double_as_longlong(fmin(z, zmax) + kM);
        else y = __double2ll_rn(z);  // integral beyond 2^53: nothing rounds up to 2^(8S-1)
        lo[q] = (uint32_t)y;
        hi[q] = (uint32_t)((unsigned long long)y >> 32);
      }
      // byte S-1-p of the four integers into one word: two byte permutes take the
      // byte from columns (0, 1) and (2, 3), a third joins the halves
#pragma unroll
      for (int p = 0; p < S; ++p) {
        const int bi = S - 1 - p, kb = bi & 3;
        const uint32_t sel = (uint32_t)(((4 + kb) << 4) | kb);
        const uint32_t s01 = bi >= 4 ? __byte_perm(hi[0], hi[1], sel) : __byte_perm(lo[0], lo[1], sel);
        const uint32_t s23 = bi >= 4 ? __byte_perm(hi[2], hi[3], sel) : __byte_perm(lo[2], lo[3], sel);
        w[p][g] = __byte_perm(s01, s23, 0x5410);
      }
    }
    uint8_t* dst = LS + oz_blk_off(row, a0, ld, 128);
#pragma unroll
    for (int p = 0; p < S; ++p)
      *reinterpret_cast<uint4*>(dst + p * slice) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  }
}

// C (n x r, column-major FP64) -> slices CS[q] of the npad x ld matrix C^T,
// blocked in tiles of Nt rows (rows k >= r and columns b >= n zero), column
// scale factors fC[k] = 2^e_k.  One warp per column k.
template <int S>
__global__ void k_oz_slice_c(const double* __restrict__ C, int n, int r, int npad, int ld, int Nt,
                             uint8_t* __restrict__ CS, double* __restrict__ fC) {
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (k >= npad) return;
  const double* ck = C + (size_t)n * k;
  double m = 0.0;
  if (k < r)
    for (int b = lane; b < n; b += 32) m = fmax(m, fabs(ck[b]));
  const int e = oz_exponent(warp_max(m));
  if (lane == 0) fC[k] = oz_pow2e(e);
  const OzScale sc = oz_scale<S>(e);
  const size_t slice = (size_t)npad * ld;
  for (int b0 = 8 * lane; b0 < ld; b0 += 256) {
    uint8_t* out = CS + oz_blk_off(k, b0, ld, Nt);
    long long y[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int b = b0 + u;
      y[u] = oz_fixed<S>((k < r && b < n) ? ck[b] : 0.0, sc);
    }
    uint2 w[S];
    oz_pack8<S>(y, w);
#pragma unroll
    for (int q = 0; q < S; ++q) *reinterpret_cast<uint2*>(out + q * slice) = w[q];
  }
}

// X (FP64, column-major: element (a, c) at X[c * xld + a], columns
// [0, kx)) -> slices of XS (ld rows x xs_row columns, blocked in 128-row
// tiles) at columns col0 + c (zero beyond kx and for rows a >= n), with the
// row exponent of xmax[a] (the largest |X| of the row, recorded by the
// half-transform), stored in eX[a].  One thread per (row a, 32-column
// chunk): consecutive threads take consecutive rows, so that a warp reads
// 256 consecutive bytes per column and writes 1 KB per slice.
template <int S>
__global__ void k_oz_slice_x(const double* __restrict__ X, int64_t xld, int n, int kx, int ld, int kblk,
                             int64_t xs_row, int64_t col0, const unsigned long long* __restrict__ xmax,
                             uint8_t* __restrict__ XS, int* __restrict__ eX) {
  const int nch = kblk / 32;
  const int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (o >= (int64_t)ld * nch) return;
  // block blockIdx.y of a launch
  X += (size_t)blockIdx.y * kx * xld;
  xmax += (size_t)blockIdx.y * ld;
  eX += (size_t)blockIdx.y * ld;
  col0 += (int64_t)blockIdx.y * kblk;
  const int ri = (int)(o & 127);
  const int64_t r2 = o >> 7;
  const int ch = (int)(r2 % nch), tile = (int)(r2 / nch);
  const int a = tile * 128 + ri;
  const int e = a < n ? oz_exponent(__longlong_as_double((long long)xmax[a])) : 0;
  if (ch == 0) eX[a] = e;
  const OzScale sc = oz_scale<S>(e);
  uint2 w[4][S];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    long long y[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int c = 32 * ch + 8 * g + u;
      y[u] = oz_fixed<S>((a < n && c < kx) ? X[(size_t)c * xld + a] : 0.0, sc);
    }
    oz_pack8<S>(y, w[g]);
  }
  const size_t slice = (size_t)ld * xs_row;
  uint8_t* out = XS + oz_blk_off(a, col0 + 32 * ch, xs_row, 128);
#pragma unroll
  for (int q = 0; q < S; ++q) {
    uint4* d = reinterpret_cast<uint4*>(out + q * slice);
    d[0] = make_uint4(w[0][q].x, w[0][q].y, w[1][q].x, w[1][q].y);
    d[1] = make_uint4(w[2][q].x, w[2][q].y, w[3][q].x, w[3][q].y);
  }
}

// xmax[a] = bits of max_c |X[c * xld + a]| (for the self-test, where X is given)
__global__ void k_row_absmax(const double* __restrict__ X, int64_t xld, int n, int kx,
                             unsigned long long* __restrict__ xmax) {
  const int a = blockIdx.x;
  double m = 0.0;
  if (a < n)
    for (int c = threadIdx.x; c < kx; c += blockDim.x) m = fmax(m, fabs(X[(size_t)c * xld + a]));
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0 && m > 0.0) atomicMax(xmax + a, (unsigned long long)__double_as_longlong(m));
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on the driver library).
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

// 8-bit tensor map over s blocked slices of a rows x kx matrix (layout of
// oz_blk_off: tiles of br rows x 32 bytes, each contiguous), as a 5D tensor
// (32 bytes, br rows, kx / 32 K steps, rows / br row tiles, s slices); a box
// is one tile of the first nbox slices, placed in shared memory one after
// another with the 32-byte swizzle.
static bool make_slice_map(CUtensorMap* m, const uint8_t* base, int64_t kx, int64_t rows, int s, int br, int nbox) {
  auto enc = tensor_map_encoder();
  if (!enc || ((uintptr_t)base & 15) || nbox < 1 || nbox > s || kx % 32 || br < 8 || br > 256 || br % 8 || rows % br) return false;
  cuuint64_t gdim[5] = {32u, (cuuint64_t)br, (cuuint64_t)(kx / 32), (cuuint64_t)(rows / br), (cuuint64_t)s};
  cuuint64_t gstr[4] = {32u, (cuuint64_t)br * 32, (cuuint64_t)(kx * br), (cuuint64_t)(kx * rows)};
  cuuint32_t box[5] = {32u, (cuuint32_t)br, 1u, 1u, (cuuint32_t)nbox}, es[5] = {1, 1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, (void*)base, gdim, gstr, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// slices that the second pass of the exchange product loads (its low diagonals)
static inline int oz_lo_slices(int s) { return std::max(1, s - std::min(s, 4)); }

static inline int rup(int x, int m) { return (x + m - 1) / m * m; }

// Column tiles of the half-transform: the widest multiple of 16 (<= 256)
// whose s accumulators fit the 512 TMEM columns (one pass per tile), then
// spread evenly over the r columns.
static void oz_col_tiles(int r, int s, int& nnt, int& Nt) {
  const int nmax = std::min(256, (512 / s) / 16 * 16);
  nnt = (r + nmax - 1) / nmax;
  Nt = rup((r + nnt - 1) / nnt, 16);
}

// Pass plan of one kind of output tile: accumulators of acc_stride TMEM
// columns, at most 512 columns; shared-memory ring of the slices 0..s-1.
static void oz_plan(OzArgs& a, int s, int Nt) {
  a.s = s;
  a.Nt = Nt;
  a.acc_stride = Nt;
  a.nd = std::min(s, 512 / a.acc_stride);
  a.b_bytes = 32 * Nt;  // the tiles of a box lie one after another (a multiple of the 256-byte swizzle atom)
  a.stage_bytes = s * (kOzABytes + a.b_bytes);
  a.stages = std::min(kOzMaxStages, (kOzSmemLimit - 1024) / a.stage_bytes);
}

// Row exponents of the handle's Cholesky vectors for squares of ld rows
// (computed once per decomposition, cached in the Cholesky state).
static const short* oz_row_exponents(Handle* h, const int* inv, int ld, cudaStream_t st) {
  ChoState* c = h->cho;
  if (const short* e = cho_lexp(c, ld)) return e;
  const int M = cho_nvec(c), n = h->nbf, vb = cho_vec_block();
  const int64_t nrs = cho_nrs(c);
  short* e = nullptr;
  if (dev_malloc(h, &e, sizeof(short) * (size_t)M * ld) != cudaSuccess) return nullptr;
  for (int J0 = 0; J0 < M; J0 += vb) {
    const int nv = std::min(vb, M - J0);
    const double* L = cho_vec_ptr(c, J0, nv, st, h);
    const int64_t rows = (int64_t)nv * ld;
    k_oz_lexp<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(inv, n, nrs, L, nv, ld, e + (size_t)J0 * ld);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (cudaGetLastError() != cudaSuccess) {
      cudaFree(e);
      return nullptr;
    }
  }
  cho_set_lexp(c, e, ld);
  return e;
}

// Per-density state of a mixed J/K batch.
struct OzDens {
  const double* C;
  int r;
  double* J;
  double* K;
  int nnt, Nt, npad, kx, kblk, nsub, ksub;
  int64_t xs_row;
  double* jrs;           // Coulomb in rs layout
  uint8_t* CS;           // slices of C
  double* fC;            // column scale factors of C
  uint8_t* XS;           // slices of X for one group of blocks
  int* eX;               // their row exponents
  CUtensorMap map_c, map_x, map_xlo;
  OzArgs ax, ak;
};

int jk_mixed(Handle* h, const double* d_C, int r, double* d_J, double* d_K, cudaStream_t st, int block, int s,
             int sk) {
  return jk_mixed_batch(h, 1, &d_C, &r, &d_J, &d_K, st, block, s, sk);
}

// J/K of k densities over one pass of the vectors: every block of vectors is
// unpacked and sliced once, the Coulomb contractions of all densities take
// one read of the block (k_vmulti), J accumulates for all densities in one
// more (k_jacc_multi), and each density runs its half-transform, X slicing and
// exchange product on the shared slices.
int jk_mixed_batch(Handle* h, int k, const double* const* Cs, const int* rs_, double* const* Js, double* const* Ks,
                   cudaStream_t st, int block, int s, int sk) {
  ChoState* c = h->cho;
  const int64_t nrs = cho_nrs(c);
  const int M = cho_nvec(c);
  const int n = h->nbf;
  if (s < 2 || s > kOzMaxSlices || sk < 2 || sk > kOzMaxSlices) {
    h->err = "mixed J/K: slices must be 2..8";
    return MG_ERR_ARG;
  }
  if (k < 1 || k > kJkMaxDens) {
    h->err = "mixed J/K: 1..8 densities per batch";
    return MG_ERR_ARG;
  }
  if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) {
    h->err = std::string("mixed J/K: error pending from earlier work: ") + cudaGetErrorString(e);
    return MG_ERR_CUDA;
  }
  for (int d = 0; d < k; ++d)
    if (!Cs[d] || !Js[d] || !Ks[d] || rs_[d] < 1) {
      h->err = "mixed J/K: a density of the batch has no factor or outputs";
      return MG_ERR_ARG;
    }
  if (M == 0) return jk_no_vectors(h, k, Js, Ks, st);
  const int ld = rup(n, 128);
  // vectors per block: one block's K extent of the exchange product, nb r
  const int nb = std::min(block, M);
  const int nblocks = (M + nb - 1) / nb;
  int G = std::min(16, nblocks);  // blocks per exchange-product group
  const int ntile = (ld / 128) * (ld / 128 + 1) / 2;
  std::vector<OzDens> dd(k);
  int kxmax = 0;
  for (int d = 0; d < k; ++d) {
    OzDens& q = dd[d];
    q.C = Cs[d];
    q.r = rs_[d];
    q.J = Js[d];
    q.K = Ks[d];
    oz_col_tiles(q.r, s, q.nnt, q.Nt);
    q.npad = q.nnt * q.Nt;
    q.kx = nb * q.r;
    q.kblk = rup(q.kx, 32);
    q.nsub = (q.kblk + kOzKChunk - 1) / kOzKChunk;
    q.ksub = rup((q.kblk + q.nsub - 1) / q.nsub, 32);
    kxmax = std::max(kxmax, q.kx);
  }
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
  const int* d_ra = cho_rs_a_dev(c);
  const int* d_rb = cho_rs_b_dev(c);
  const int* inv = cho_inv_dev(c);
  const size_t nn = (size_t)n * n;
  // blocks per launch of the slicing, the half-transform and the Coulomb part: a
  // power of two (storage blocks of 1024 vectors are not straddled), as many as
  // keep the sliced squares within 512 MB and X within 256 MB.  One block of 64
  // vectors is less than two waves of half-transform tiles below 500 functions and
  // a few microseconds below 150.  Keeping the squares in L2 (128 MB) instead is
  // slower: 403 functions, two densities 6.66 ms with single blocks, 6.70 with 128
  // MB, 5.30 with 512; 96 functions 562, 257, 255 us; 168 functions 977, 588, 458 us.
  int Lg = 1;
  while (2 * Lg <= 16 && Lg < nblocks && (size_t)2 * Lg * s * nb * ld * ld <= kOzGroupBytes &&
         (size_t)2 * Lg * 8 * ld * kxmax <= ((size_t)256 << 20))
    Lg *= 2;
  // Memory short: half as many blocks per launch, then per group of the exchange
  // product, until the workspace can be had (one block each is the least).
  int nbg = 0, jsplit = 0;
  size_t need = 0;
  char* ws = nullptr;
  for (;;) {
    nbg = nb * Lg;
    jsplit = jacc_splits(nrs, nbg, nsm);
    // one term per take() below (each rounded up to 256 bytes)
    need = 8 * (size_t)nbg * k + (size_t)s * nbg * ld * ld + 4 * (size_t)nbg * ld + 8 * (size_t)ld * kxmax * Lg +
           8 * (size_t)ld * Lg + 8 * (size_t)nsm * 128 * 128 + sizeof(int) +
           8 * (size_t)(jsplit * (size_t)nrs + vmulti_ranges(nrs) * (size_t)nbg) * k + 10 * 256;
    for (OzDens& q : dd) {
      q.xs_row = (int64_t)G * q.kblk;
      need += 8 * (size_t)nrs + (size_t)s * q.npad * ld + 8 * (size_t)q.npad + (size_t)sk * ld * q.xs_row +
              4 * (size_t)G * ld + 6 * 256;
    }
    ws = (char*)ws_get(h, need, st);
    if (ws || (Lg == 1 && G == 1)) break;
    if (Lg > 1) Lg /= 2;
    else G = (G + 1) / 2;
  }
  if (!ws) { h->err = "jk workspace allocation failed"; return MG_ERR_MEMORY; }
  char* const ws_end = ws + need;
  auto take = [&](size_t bytes) { char* p = ws; ws += (bytes + 255) & ~(size_t)255; return (void*)p; };
  double* V = (double*)take(8 * (size_t)nbg * k);  // V[d nbg + J]
  uint8_t* LS = (uint8_t*)take((size_t)s * nbg * ld * ld);
  int* eA = (int*)take(4 * (size_t)nbg * ld);
  double* Xf = (double*)take(8 * (size_t)ld * kxmax * Lg);  // column-major, ld rows
  unsigned long long* xmax = (unsigned long long*)take(8 * (size_t)ld * Lg);
  double* P = (double*)take(8 * (size_t)nsm * 128 * 128);
  int* d_err = (int*)take(sizeof(int));
  double* jrs_all = (double*)take(8 * (size_t)nrs * k * jsplit);  // jrs of density d at d nrs, per split
  double* Vp = (double*)take(8 * (size_t)vmulti_ranges(nrs) * nbg * k);
  double* dws = (double*)take(8 * (size_t)nrs * k);      // packed weighted densities
  for (int d = 0; d < k; ++d) {
    OzDens& q = dd[d];
    q.jrs = jrs_all + (size_t)d * nrs;
    q.CS = (uint8_t*)take((size_t)s * q.npad * ld);
    q.fC = (double*)take(8 * (size_t)q.npad);
    q.XS = (uint8_t*)take((size_t)sk * ld * q.xs_row);
    q.eX = (int*)take(4 * (size_t)G * ld);
  }
  if (ws > ws_end) { h->err = "mixed J/K: workspace layout exceeds its size"; return MG_ERR_CUDA; }
  // every launch is checked at once, so that an error names its kernel
  auto launched = [&](const char* what) {
    g_launches.fetch_add(1, std::memory_order_relaxed);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return true;
    h->err = std::string("mixed J/K: ") + what + ": " + cudaGetErrorString(e);
    return false;
  };
  CUtensorMap map_l;
  if (!make_slice_map(&map_l, LS, ld, (int64_t)nbg * ld, s, 128, s)) {
    h->err = "tensor maps for the exchange GEMMs could not be encoded";
    return MG_ERR_CUDA;
  }
  for (OzDens& q : dd)
    if (!make_slice_map(&q.map_c, q.CS, ld, q.npad, s, q.Nt, s) ||
        !make_slice_map(&q.map_x, q.XS, q.xs_row, ld, sk, 128, sk) ||
        !make_slice_map(&q.map_xlo, q.XS, q.xs_row, ld, sk, 128, oz_lo_slices(sk))) {
      h->err = "tensor maps for the exchange GEMMs could not be encoded";
      return MG_ERR_CUDA;
    }
  bool attr = true;
  oz_with_slices(s, [&](auto S) { attr &= smem_attr_once((const void*)oz_gemm_kernel<false, decltype(S)::value>, kOzSmemLimit); });
  oz_with_slices(sk, [&](auto S) { attr &= smem_attr_once((const void*)oz_gemm_kernel<true, decltype(S)::value>, kOzSmemLimit); });
  if (!attr) {
    h->err = "exchange GEMMs: shared-memory limit could not be raised";
    return MG_ERR_CUDA;
  }
  for (OzDens& q : dd) {
    OzArgs& ax = q.ax;
    OzArgs& ak = q.ak;
    ax = OzArgs{};
    ak = OzArgs{};
    oz_plan(ax, s, q.Nt);
    oz_plan(ak, sk, 128);
    if (ax.stages < 2 || ak.stages < 2) { h->err = "mixed J/K: slice tiles do not fit in shared memory"; return MG_ERR_ARG; }
    ax.err = ak.err = d_err;
    ax.nrt = ld / 128; ax.nnt = q.nnt; ax.ld = ld; ax.kx = rup(n, kOzCutCols); ax.n = n; ax.r = q.r; ax.eA = eA; ax.fB = q.fC; ax.X = Xf;
    ax.xld = ld; ax.xmax = xmax; ax.jx = nb;
    ak.ld = ld; ak.n = n; ak.ntile = ntile; ak.nsub = q.nsub; ak.kblk = q.kblk; ak.ksub = q.ksub; ak.eX = q.eX;
    ak.P = P; ak.K = q.K;
  }
  if (cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess ||
      cudaMemsetAsync(jrs_all, 0, 8 * (size_t)nrs * k * jsplit, st) != cudaSuccess) {
    h->err = std::string("mixed J/K: clearing buffers: ") + cudaGetErrorString(cudaGetLastError());
    return MG_ERR_CUDA;
  }
  for (int d = 0; d < k; ++d) {
    OzDens& q = dd[d];
    if (cudaMemsetAsync(q.K, 0, 8 * nn, st) != cudaSuccess) {
      h->err = std::string("mixed J/K: clearing K: ") + cudaGetErrorString(cudaGetLastError());
      return MG_ERR_CUDA;
    }
    k_density_rs<<<nb256(nrs), 256, 0, st>>>(d_ra, d_rb, nrs, q.C, n, q.r, dws + (size_t)d * nrs);
    if (!launched("k_density_rs")) return MG_ERR_CUDA;
  }
  const short* eL = oz_row_exponents(h, inv, ld, st);
  if (!eL) { h->err = "mixed J/K: row exponents could not be stored"; return MG_ERR_MEMORY; }
  for (OzDens& q : dd) {
    oz_with_slices(s, [&](auto S) {
      k_oz_slice_c<decltype(S)::value><<<(q.npad + 7) / 8, 256, 0, st>>>(q.C, n, q.r, q.npad, ld, q.Nt, q.CS, q.fC);
    });
    if (!launched("k_oz_slice_c")) return MG_ERR_CUDA;
  }
  for (int g0 = 0; g0 < nblocks; g0 += G) {
    const int gn = std::min(G, nblocks - g0);
    for (int bi = 0; bi < gn; bi += Lg) {
      const int bn = std::min(Lg, gn - bi);
      const int J0 = (g0 + bi) * nb;
      const int nv = std::min(bn * nb, M - J0);
      const double* Lb = cho_vec_ptr(c, J0, nv, st, h);
      if (!Lb) { h->err = "vector block straddles storage blocks"; return MG_ERR_ARG; }
      oz_with_slices(s, [&](auto S) {
        k_oz_slice_l<decltype(S)::value>
            <<<dim3(ld / kOzCutRows, (n + kOzCutCols - 1) / kOzCutCols, (nv + kOzVecs - 1) / kOzVecs), 2 * kOzCutRows, 0, st>>>(
                inv, n, nrs, Lb, nv, ld, (int64_t)nbg * ld * ld, eL + (size_t)J0 * ld, LS, eA);
      });
      if (!launched("k_oz_slice_l")) return MG_ERR_CUDA;
      launch_vmulti(Lb, nrs, nv, nbg, k, dws, Vp, V, st);
      if (!launched("k_vmulti")) return MG_ERR_CUDA;
      launch_jacc(Lb, nrs, nv, nbg, k, jsplit, V, jrs_all, st);
      if (!launched("k_jacc_multi")) return MG_ERR_CUDA;
      for (OzDens& q : dd) {
        // a short last block: clear the columns of the missing vectors
        if (nv < bn * nb)
          cudaMemsetAsync(Xf + (size_t)nv * q.r * ld, 0, 8 * (size_t)(bn * nb - nv) * q.r * ld, st);
        cudaMemsetAsync(xmax, 0, 8 * (size_t)ld * bn, st);
        // X_J = L_J C for the blocks (the slice map covers nbg vectors; nv <= nbg of them are used)
        OzArgs& ax = q.ax;
        ax.nJ = nv;
        ax.nitems = ax.nrt * nv * q.nnt;
        const int gx = std::min(ax.nitems, nsm);
        oz_with_slices(s, [&](auto S) {
          oz_gemm_kernel<false, decltype(S)::value><<<gx, kOzThreads, ax.stages * ax.stage_bytes + 1024, st>>>(
              map_l, q.map_c, map_l, ax);
        });
        if (!launched("oz_gemm_kernel<false>")) return MG_ERR_CUDA;
        oz_with_slices(sk, [&](auto S) {
          k_oz_slice_x<decltype(S)::value><<<dim3(nb256((int64_t)ld * (q.kblk / 32)), bn), 256, 0, st>>>(
              Xf, ld, n, q.kx, ld, q.kblk, q.xs_row, (int64_t)bi * q.kblk, xmax, q.XS, q.eX + (size_t)bi * ld);
        });
        if (!launched("k_oz_slice_x")) return MG_ERR_CUDA;
      }
    }
    // K += X X^T over the group (lower tiles), per density
    for (OzDens& q : dd) {
      OzArgs& ak = q.ak;
      ak.nblk = gn;
      ak.nitems = ntile * gn * q.nsub;
      const int gk = std::min(ak.nitems, nsm);
      oz_with_slices(sk, [&](auto S) {
        oz_gemm_kernel<true, decltype(S)::value><<<gk, kOzThreads, ak.stages * ak.stage_bytes + 1024, st>>>(
            q.map_x, q.map_x, q.map_xlo, ak);
      });
      if (!launched("oz_gemm_kernel<true>")) return MG_ERR_CUDA;
    }
  }
  for (OzDens& q : dd) {
    k_symmetrize_lower<<<nb256((int64_t)nn), 256, 0, st>>>(q.K, n);
    if (!launched("k_symmetrize_lower")) return MG_ERR_CUDA;
    k_finish_j<<<nb256((int64_t)nn), 256, 0, st>>>(inv, q.jrs, jsplit, (int64_t)k * nrs, n, q.J);
    if (!launched("k_finish_j")) return MG_ERR_CUDA;
  }
  if (const cudaError_t e = cudaGetLastError(); e != cudaSuccess) {
    h->err = std::string("mixed J/K: ") + cudaGetErrorString(e);
    return MG_ERR_CUDA;
  }
  int herr = 0;
  cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (const cudaError_t e = cudaStreamSynchronize(st); e != cudaSuccess) {
    h->err = std::string("mixed J/K: ") + cudaGetErrorString(e);
    return MG_ERR_CUDA;
  }
  if (herr) {
    h->err = "exchange GEMMs: a pipeline wait ran out (result incomplete)";
    return MG_ERR_CUDA;
  }
  return 0;
}

// The sliced engine on given dense matrices (verification of the kernels
// used by jk_mixed): X = A B (A: ld x ld, B: ld x r, X: ld x r, all
// column-major) and K = X X^T (lower triangle, column-major ld x ld).
int oz_selftest(Handle* h, int ld, int r, int s, const double* d_A, const double* d_B, double* d_X, double* d_K,
                uint8_t* d_slices, int* d_exps, cudaStream_t st) {
  if (ld < 128 || ld % 128 || r < 1 || s < 2 || s > kOzMaxSlices) return MG_ERR_ARG;
  int nnt, Nt;
  oz_col_tiles(r, s, nnt, Nt);
  const int npad = nnt * Nt;
  const int kblk = rup(r, 32);
  const int nsub = (kblk + kOzKChunk - 1) / kOzKChunk;
  const int ksub = rup((kblk + nsub - 1) / nsub, 32);
  int nsm = 148;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, h->device);
  const size_t need = (size_t)s * ld * ld + 4 * (size_t)ld + (size_t)s * npad * ld + 8 * (size_t)npad +
                      (size_t)s * ld * kblk + 4 * (size_t)ld + 16 * (size_t)ld + 8 * (size_t)nsm * 128 * 128 +
                      18 * 256;
  char* ws = (char*)ws_get(h, need, st);
  if (!ws) return MG_ERR_MEMORY;
  auto take = [&](size_t bytes) { char* p = ws; ws += (bytes + 255) & ~(size_t)255; return (void*)p; };
  uint8_t* LS = (uint8_t*)take((size_t)s * ld * ld);
  int* eA = (int*)take(4 * (size_t)ld);
  uint8_t* CS = (uint8_t*)take((size_t)s * npad * ld);
  double* fC = (double*)take(8 * (size_t)npad);
  uint8_t* XS = (uint8_t*)take((size_t)s * ld * kblk);
  int* eX = (int*)take(4 * (size_t)ld);
  unsigned long long* amax = (unsigned long long*)take(8 * (size_t)ld);
  unsigned long long* xmax = (unsigned long long*)take(8 * (size_t)ld);
  double* P = (double*)take(8 * (size_t)nsm * 128 * 128);
  int* d_err = (int*)take(sizeof(int));
  CUtensorMap map_l, map_c, map_x, map_xlo;
  if (!make_slice_map(&map_l, LS, ld, ld, s, 128, s) || !make_slice_map(&map_c, CS, ld, npad, s, Nt, s) ||
      !make_slice_map(&map_x, XS, kblk, ld, s, 128, s) ||
      !make_slice_map(&map_xlo, XS, kblk, ld, s, 128, oz_lo_slices(s)))
    return MG_ERR_CUDA;
  OzArgs ax{}, ak{};
  oz_plan(ax, s, Nt);
  oz_plan(ak, s, 128);
  bool attr = true;
  oz_with_slices(s, [&](auto S) {
    attr &= smem_attr_once((const void*)oz_gemm_kernel<false, decltype(S)::value>, kOzSmemLimit) &&
            smem_attr_once((const void*)oz_gemm_kernel<true, decltype(S)::value>, kOzSmemLimit);
  });
  if (!attr) return MG_ERR_CUDA;
  ax.err = ak.err = d_err;
  ax.nrt = ld / 128; ax.nnt = nnt; ax.ld = ax.kx = ld; ax.n = ld; ax.r = r; ax.eA = eA; ax.fB = fC; ax.X = d_X; ax.xld = ld;
  ax.xmax = xmax; ax.jx = 1; ax.nJ = 1; ax.nitems = ax.nrt * nnt;
  ak.ld = ld; ak.n = ld; ak.ntile = (ld / 128) * (ld / 128 + 1) / 2; ak.nsub = nsub; ak.kblk = kblk; ak.ksub = ksub;
  ak.eX = eX; ak.P = P; ak.K = d_K; ak.nblk = 1; ak.nitems = ak.ntile * nsub;
  cudaMemsetAsync(d_err, 0, sizeof(int), st);
  cudaMemsetAsync(d_K, 0, 8 * (size_t)ld * ld, st);
  cudaMemsetAsync(amax, 0, 8 * (size_t)ld, st);
  cudaMemsetAsync(xmax, 0, 8 * (size_t)ld, st);
  k_row_absmax<<<ld, 256, 0, st>>>(d_A, ld, ld, ld, amax);
  oz_with_slices(s, [&](auto S) {
    k_oz_slice_x<decltype(S)::value><<<nb256((int64_t)ld * (ld / 32)), 256, 0, st>>>(d_A, ld, ld, ld, ld, ld, ld, 0,
                                                                                    amax, LS, eA);
  });
  if (d_slices) cudaMemcpyAsync(d_slices, LS, (size_t)s * ld * ld, cudaMemcpyDeviceToDevice, st);
  if (d_exps) cudaMemcpyAsync(d_exps, eA, 4 * (size_t)ld, cudaMemcpyDeviceToDevice, st);
  oz_with_slices(s, [&](auto S) {
    k_oz_slice_c<decltype(S)::value><<<(npad + 7) / 8, 256, 0, st>>>(d_B, ld, r, npad, ld, Nt, CS, fC);
  });
  oz_with_slices(s, [&](auto S) {
    oz_gemm_kernel<false, decltype(S)::value>
        <<<std::min(ax.nitems, nsm), kOzThreads, ax.stages * ax.stage_bytes + 1024, st>>>(map_l, map_c, map_l, ax);
  });
  oz_with_slices(s, [&](auto S) {
    k_oz_slice_x<decltype(S)::value><<<nb256((int64_t)ld * (kblk / 32)), 256, 0, st>>>(d_X, ld, ld, r, ld, kblk, kblk,
                                                                                      0, xmax, XS, eX);
  });
  oz_with_slices(s, [&](auto S) {
    oz_gemm_kernel<true, decltype(S)::value>
        <<<std::min(ak.nitems, nsm), kOzThreads, ak.stages * ak.stage_bytes + 1024, st>>>(map_x, map_x, map_xlo, ak);
  });
  g_launches.fetch_add(6, std::memory_order_relaxed);
  if (cudaGetLastError() != cudaSuccess) return MG_ERR_CUDA;
  int herr = 0;
  cudaMemcpyAsync(&herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess) return MG_ERR_CUDA;
  return herr ? MG_ERR_CUDA : 0;
}

}  // namespace mg
