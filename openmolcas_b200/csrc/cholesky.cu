// Pivoted Cholesky decomposition of the ERI matrix on the GPU with the
// semantics of OpenMolcas's default algorithm 4 (cholesky_util):
//
//   pass loop  CHO_DECDRV          cho_decdrv.F90:98-260
//   SetPass    max diag, DiaMin    cho_setpass.F90:29-47
//   GetMaxShl  one shell pair      cho_getmaxshl.F90, MXSHPR=1 (cho_inp.F90:709-715)
//   Qualify_2  diag >= DiaMin      cho_qualify_2.F90 (IALQUA = 2, cho_inp.F90:156), MaxQual = 100
//   columns    (CD|AB) all CD      cho_mca_calcint_1.F90 + PLF_Cho
//   Dec_Qual   Q = MQ - LQ LQ^T    cho_dec_qual.F90:57-83 (Thr = max(ThrCom, Dmax Span))
//   CD_InCore_1p pivot rule        cd_incore_1p.F90:33-85 (Acc tie rule, host FP64)
//   Subtr      X -= L LQ^T         cho_vecbuf_subtr.F90:188-215
//   CompVec    scale/diag update   cho_compvec.F90:40-120 + Cho_ChkDia_A4
//   SetRed     damped screening    cho_setred.F90:72-100 (MODE_SCREEN 1)
//
// Device work: ERI diagonal and columns (eri.cu kernels), the reduced set and
// the choice of shell pair, the qualified block, and one fused kernel for the
// new vectors.  Host work per pass: the qualification list, the work items and
// the in-core CD of the <=100 x 100 qualified block (sequential, exact
// reference semantics); it waits for the device twice (the chosen pair, the
// qualified block).  Vectors are FP64 in reduced-set ("rs") layout, blocks of
// kVecBlock columns.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "cho_qualify.h"
#include "kern_common.cuh"
#include "mg_internal.h"

namespace mg {

constexpr int kVecBlock = 1024;  // vectors per storage block
// largest buffer of a decomposition that the handle keeps for the next one
constexpr size_t kKeepBytes = (size_t)256 << 20;

// ------------------------------------------------------------------ kernels
// rs descriptor: AO pair (a,b) with its shell pair and local indices
struct RsDev {
  int sp;          // shell pair id
  short ma, ka;    // component and contracted index of a in its shell
  short mb, kb;    // same for b
};

// diag[t] = (ab|ab) from the diagonal quartet blocks
__global__ void k_extract_diag(const RsDev* __restrict__ rs, int64_t nrs, const DPair* __restrict__ pairs,
                               const int64_t* __restrict__ blk_off, const double* __restrict__ blk,
                               double* __restrict__ diag) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nrs) return;
  const RsDev r = rs[t];
  const DPair& P = pairs[r.sp];
  const int nij = P.nci * P.ncj;
  const int ij = r.ka + P.nci * r.kb;
  const int64_t ijkl = ij + (int64_t)nij * ij;
  const int64_t nijkl = (int64_t)nij * nij;
  const int sab = r.ma + P.nsa * r.mb;
  const int nsab = P.nsa * P.nsb;
  diag[t] = blk[blk_off[r.sp] + ijkl + nijkl * (sab + (int64_t)nsab * sab)];
}

// Element (row | col) of the (CD|AB) block of row's shell pair (Eval_IJKL
// layout); col belongs to the ket pair A.
__device__ __forceinline__ double cho_blk(const double* __restrict__ blk, const RsDev& r, const DPair& C, const RsDev& c,
                                          const DPair& A) {
  const int nij = C.nci * C.ncj, nijkl = nij * A.nci * A.ncj;
  return __ldg(blk + r.ka + C.nci * r.kb + (int64_t)nij * (c.ka + A.nci * c.kb) +
               (int64_t)nijkl * (r.ma + C.nsa * r.mb + (int64_t)C.nsa * C.nsb * (c.ma + A.nsa * c.mb)));
}

// One warp per shell pair: Cho_SetRed mode 1 of the pass just done (no abs:
// keep diag > 0 with sqrt(diag xm) damp > thrcom, xm the largest |diagonal|,
// nothing once xm <= thrcom; apply = 0 before the first pass), then the
// pair's maxima (CHO_SETMAXSHL): diash[sp] = max(0, largest diagonal) over its
// members in the reduced set, -1 when none is in it, diash[nsp + sp] their
// largest |diagonal|; alive[sp] = some member is in the reduced set.
__global__ void k_cho_scan(const double* __restrict__ diag, unsigned char* __restrict__ inred,
                           const int64_t* __restrict__ sp_first, const int* __restrict__ sp_count, int nsp,
                           const unsigned long long* __restrict__ xmbits, int apply, double damp, double thrcom,
                           double* __restrict__ diash, unsigned char* __restrict__ alive) {
  const int sp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (sp >= nsp) return;
  const double xm = __longlong_as_double((long long)*xmbits);
  const bool conv = !(xm > thrcom);
  double m = -1.0, ma = 0.0;
  const int64_t f = sp_first[sp];
  for (int i = lane; i < sp_count[sp]; i += 32) {
    if (!inred[f + i]) continue;
    const double d = diag[f + i];
    if (apply && (conv || !(d > 0.0 && sqrt(d * xm) * damp > thrcom))) {
      inred[f + i] = 0;
      continue;
    }
    m = fmax(m, fmax(d, 0.0));
    ma = fmax(ma, fabs(d));
  }
  for (int o = 16; o > 0; o >>= 1) {
    m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    ma = fmax(ma, __shfl_xor_sync(0xffffffffu, ma, o));
  }
  if (lane == 0) {
    diash[sp] = m;
    diash[nsp + sp] = ma;
    alive[sp] = m >= 0.0;
  }
}

// What the host reads once per pass, at the head of one buffer: then the
// diagonals (maxcnt doubles) and reduced-set flags (maxcnt bytes) of the chosen
// shell pair and alive[nsp].
struct ChoSel {
  double dgmax, smax;  // largest |diagonal|; the chosen pair's maximum
  int spab, flags;     // the chosen pair; error flags of the update kernel
  long long pad;
};

// Cho_SetPass / Cho_GetMaxShl: the largest |diagonal|, and the shell pair of
// the largest diagonal above thrcom (the first of equal ones; diagonals at or
// below thrcom count as 0).  One CTA; clears xm for the next pass.
__global__ void __launch_bounds__(1024) k_cho_select(const double* __restrict__ diash, int nsp, double thrcom,
                                                     const int64_t* __restrict__ sp_first,
                                                     const int* __restrict__ sp_count, const double* __restrict__ diag,
                                                     const unsigned char* __restrict__ inred,
                                                     const int* __restrict__ flags, unsigned long long* __restrict__ xm,
                                                     ChoSel* __restrict__ sel, double* __restrict__ dpair,
                                                     unsigned char* __restrict__ rpair) {
  __shared__ double sg[32], sv[32];
  __shared__ int si[32];
  double g = 0.0, v = -1.0;
  int idx = 0x7fffffff;
  for (int sp = threadIdx.x; sp < nsp; sp += blockDim.x) {
    const double x = diash[sp] > thrcom ? diash[sp] : 0.0;
    if (x > v) { v = x; idx = sp; }
    g = fmax(g, diash[nsp + sp]);
  }
  auto join = [&](double g2, double v2, int i2) {
    g = fmax(g, g2);
    if (v2 > v || (v2 == v && i2 < idx)) { v = v2; idx = i2; }
  };
  for (int o = 16; o > 0; o >>= 1) {
    const double g2 = __shfl_xor_sync(0xffffffffu, g, o), v2 = __shfl_xor_sync(0xffffffffu, v, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
    join(g2, v2, i2);
  }
  if ((threadIdx.x & 31) == 0) {
    sg[threadIdx.x >> 5] = g;
    sv[threadIdx.x >> 5] = v;
    si[threadIdx.x >> 5] = idx;
  }
  __syncthreads();
  for (int w = 0; w < (int)(blockDim.x >> 5); ++w) join(sg[w], sv[w], si[w]);
  if (threadIdx.x == 0) {
    sel->dgmax = g;
    sel->smax = v;
    sel->spab = idx;
    sel->flags = *flags;
    *xm = 0;
  }
  const int64_t f = sp_first[idx];
  for (int i = threadIdx.x; i < sp_count[idx]; i += blockDim.x) {
    dpair[i] = diag[f + i];
    rpair[i] = inred[f + i];
  }
}

// LQ: the rows of the previous vectors at the nq qualified AO pairs,
// lq[J nq + i] = L[rows[i], J], and this CTA's share of LQ LQ^T (lower
// triangle, jb vectors at a time, in part[blockIdx.x nq^2 ..]).  Lt: the
// storage blocks of kVecBlock vectors.
__global__ void __launch_bounds__(256) k_cho_lq(const double* const* __restrict__ Lt, int64_t nrs, int M,
                                                const int* __restrict__ rows, int nq, int jb,
                                                double* __restrict__ lq, double* __restrict__ part) {
  extern __shared__ double cq_sl[];  // jb x nq
  double* pb = part + (size_t)blockIdx.x * nq * nq;
  bool first = true;
  for (int j0 = blockIdx.x * jb; j0 < M; j0 += gridDim.x * jb, first = false) {
    const int nj = min(jb, M - j0);
    for (int o = threadIdx.x; o < nj * nq; o += blockDim.x) {
      const int jj = o / nq, i = o - jj * nq, J = j0 + jj;
      const double v = Lt[J / kVecBlock][rows[i] + nrs * (J % kVecBlock)];
      cq_sl[o] = v;
      lq[(size_t)J * nq + i] = v;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < nq * nq; o += blockDim.x) {
      const int j = o / nq, i = o - j * nq;
      if (i < j) continue;
      double s = first ? 0.0 : pb[o];
      for (int jj = 0; jj < nj; ++jj) s = fma(cq_sl[jj * nq + i], cq_sl[jj * nq + j], s);
      pb[o] = s;
    }
    __syncthreads();
  }
}

// Cho_Dec_Qual: Q = MQ - LQ LQ^T, MQ the integrals among the qualified AO
// pairs (all of shell pair spab), the shares summed in a fixed order.
__global__ void k_cho_q(const RsDev* __restrict__ rs, const DPair* __restrict__ pairs,
                        const double* __restrict__ blk, const int* __restrict__ rows, int nq, int spab,
                        const double* __restrict__ part, int nparts, double* __restrict__ Q) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= nq * nq) return;
  const int j = o / nq, i = o - j * nq;
  const DPair& A = pairs[spab];
  const RsDev r = rs[rows[i]], c = rs[rows[j]];
  const size_t lo = i >= j ? (size_t)j * nq + i : (size_t)i * nq + j;
  double s = 0.0;
  for (int p = 0; p < nparts; ++p) s += part[(size_t)p * nq * nq + lo];
  Q[o] = cho_blk(blk, r, A, c, A) - s;
}

// Cho_Subtr and Cho_CompVec of one pass, for the pivots i0 .. i0 + ni (at most
// 32 at a time; later launches count the earlier pivots' vectors as previous
// ones, their LQ rows being those of K):
//   k_cho_subtr    s_i = sum_J L[t, J] LQ[i, J] over a range of the previous
//                  vectors (blockIdx.y), two rows per thread, into part[range]
//   k_cho_compvec  gather the integral columns straight from the ERI blocks,
//                  x_i -= s_i (the ranges in order), scale, diagonal update,
//                  Cho_ChkDia_A4, x_j -= K_ji x_i, and store the new columns
// Rows are independent: the reference's per-vector steps touch each row only
// through its own diagonal.  Rows outside the reduced set read nothing and get
// zeros.  The previous vectors are the only large operand, read once against
// NK FMAs per element, so HBM bounds k_cho_subtr up to NK = 16 and the FP64 pipe
// above; the ranges are there for small systems, whose rows alone neither fill
// the chip nor hide the latency of one serial pass over the vectors.
// par: fac[nk] | K[nk x nk] (column i: vector i); ipar: qrs[nk] | colsel[nk].
constexpr int kUpdThreads = 128;
constexpr int kUpdRows = 2 * kUpdThreads;  // rows per CTA of k_cho_subtr
constexpr int kUpdJ = 32;                  // vectors per shared-memory chunk (divides kVecBlock)

struct ChoUpd {
  double* const* Lt;
  int64_t nrs;
  int M, i0, ni, nk, nq, spab, last;
  int jper, nrange;     // previous vectors per range (a multiple of kUpdJ), ranges
  double* part;         // [range][i][nrs]
  const double* lq;
  const double* blk;
  const int64_t* base;  // first element of a shell pair's bra block (times ksz)
  int64_t ksz;          // elements of the ket block
  const RsDev* rs;
  const DPair* pairs;
  const unsigned char* inred;
  double* diag;
  const double* par;
  const int* ipar;
  double qdmax, damp, thrcom, thrneg, tooneg;
  int* flags;
  unsigned long long* xm;
};

template <int NK>
__global__ void __launch_bounds__(kUpdThreads) k_cho_subtr(const ChoUpd u) {
  constexpr int KV = (kUpdJ * NK + kUpdThreads - 1) / kUpdThreads;  // LQ values a thread stages
  __shared__ __align__(16) double sl[2][kUpdJ][NK];
  __shared__ int ssel[NK];
  const int tid = threadIdx.x;
  const int64_t t0 = blockIdx.x * (int64_t)kUpdRows + tid, t1 = t0 + kUpdThreads;
  const bool a0 = t0 < u.nrs && u.inred[t0], a1 = t1 < u.nrs && u.inred[t1];
  if (tid < NK) ssel[tid] = tid < u.ni ? u.ipar[u.nk + u.i0 + tid] : 0;
  const int jb = blockIdx.y * u.jper, je = min(u.M + u.i0, jb + u.jper);
  if (!__syncthreads_or(a0 || a1)) return;
  double acc[2][NK], lqv[KV];
#pragma unroll
  for (int i = 0; i < NK; ++i) acc[0][i] = acc[1][i] = 0.0;
  auto stage = [&](int j0) {
#pragma unroll
    for (int v = 0; v < KV; ++v) {
      const int o = tid + v * kUpdThreads, jj = o / NK, i = o - jj * NK;
      lqv[v] = (o < kUpdJ * NK && j0 + jj < je && i < u.ni) ? __ldg(u.lq + (size_t)(j0 + jj) * u.nq + ssel[i]) : 0.0;
    }
  };
  // eight vectors of both rows are in flight while the eight before them are used
  double x0[8], x1[8];
  auto load = [&](int j) {
    const double* Lp = u.Lt[j / kVecBlock] + u.nrs * (j % kVecBlock);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const double* p = Lp + u.nrs * e;
      x0[e] = a0 && j + e < je ? __ldg(p + t0) : 0.0;
      x1[e] = a1 && j + e < je ? __ldg(p + t1) : 0.0;
    }
  };
  stage(jb);
  if (jb < je) load(jb);
  int s = 1;
  for (int j = jb; j < je; j += 8) {
    const int q = (j - jb) % kUpdJ;
    if (q == 0) {
      s ^= 1;
      double* sf = &sl[s][0][0];
#pragma unroll
      for (int v = 0; v < KV; ++v)
        if (tid + v * kUpdThreads < kUpdJ * NK) sf[tid + v * kUpdThreads] = lqv[v];
      __syncthreads();
      if (j + kUpdJ < je) stage(j + kUpdJ);
    }
    double y0[8], y1[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      y0[e] = x0[e];
      y1[e] = x1[e];
    }
    if (j + 8 < je) load(j + 8);
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int i = 0; i < NK; ++i) {
        const double l = sl[s][q + e][i];
        acc[0][i] = fma(y0[e], l, acc[0][i]);
        acc[1][i] = fma(y1[e], l, acc[1][i]);
      }
  }
  double* p = u.part + (size_t)blockIdx.y * u.ni * u.nrs;
#pragma unroll
  for (int i = 0; i < NK; ++i) {
    if (i >= u.ni) break;
    if (a0) p[(size_t)i * u.nrs + t0] = acc[0][i];
    if (a1) p[(size_t)i * u.nrs + t1] = acc[1][i];
  }
}

template <int NK>
__global__ void __launch_bounds__(kUpdThreads) k_cho_compvec(const ChoUpd u) {
  __shared__ double sK[NK * NK], sfac[NK], smax[kUpdThreads / 32];
  __shared__ int sq[NK];
  const int tid = threadIdx.x;
  const int64_t t = blockIdx.x * (int64_t)kUpdThreads + tid;
  const bool act = t < u.nrs && u.inred[t];
  for (int o = tid; o < NK; o += kUpdThreads) {
    const bool ok = o < u.ni;
    sfac[o] = ok ? u.par[u.i0 + o] : 0.0;
    sq[o] = ok ? u.ipar[u.i0 + o] : -1;
  }
  for (int o = tid; o < NK * NK; o += kUpdThreads) {
    const int j = o % NK, i = o / NK;
    sK[o] = (i < u.ni && j < u.ni) ? u.par[u.nk + (size_t)u.nk * (u.i0 + i) + u.i0 + j] : 0.0;
  }
  __syncthreads();
  double acc[NK];
#pragma unroll
  for (int i = 0; i < NK; ++i) acc[i] = 0.0;
  if (act) {
    for (int r = 0; r < u.nrange; ++r)
#pragma unroll
      for (int i = 0; i < NK; ++i)
        if (i < u.ni) acc[i] += __ldg(u.part + ((size_t)r * u.ni + i) * u.nrs + t);
    const RsDev rt = u.rs[t];
    const DPair& C = u.pairs[rt.sp];
    const DPair& A = u.pairs[u.spab];
    const double* b = u.blk + u.base[rt.sp] * u.ksz;
#pragma unroll
    for (int i = 0; i < NK; ++i)
      if (i < u.ni) acc[i] = cho_blk(b, rt, C, u.rs[sq[i]], A) - acc[i];
  }
  double dabs = 0.0;
  if (t < u.nrs) {
    double d = act ? u.diag[t] : 0.0;
    const int Mp = u.M + u.i0;
#pragma unroll
    for (int i = 0; i < NK; ++i) {
      if (i >= u.ni) break;
      double x = 0.0;
      if (act) {
        x = acc[i] * sfac[i];
        if (d == 0.0) x = 0.0;
        d -= x * x;
        if (t == sq[i]) d = 0.0;  // Cho_P_ZeroDiag
        if (d < 0.0 && d < u.thrneg) {  // Cho_ChkDia_A4
          if (d < u.tooneg) atomicOr(u.flags, 1);
          d = 0.0;
        }
        if (sqrt(fabs(d) * u.qdmax) * u.damp <= u.thrcom) d = 0.0;
#pragma unroll
        for (int j = 0; j < NK; ++j)
          if (j > i) acc[j] -= sK[j + NK * i] * x;
      }
      const int c = Mp + i;
      u.Lt[c / kVecBlock][t + u.nrs * (c % kVecBlock)] = x;
    }
    if (act) {
      u.diag[t] = d;
      dabs = fabs(d);
    }
  }
  if (u.last) {  // the largest |diagonal| left (a maximum: independent of the order)
    for (int o = 16; o > 0; o >>= 1) dabs = fmax(dabs, __shfl_xor_sync(0xffffffffu, dabs, o));
    if ((tid & 31) == 0) smax[tid >> 5] = dabs;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < kUpdThreads / 32; ++w) dabs = fmax(dabs, smax[w]);
      if (dabs > 0.0) atomicMax(u.xm, (unsigned long long)__double_as_longlong(dabs));
    }
  }
}

// ranges of the previous vectors: about 6 CTAs per SM in all, at least 64
// vectors each
static int upd_ranges(int64_t nrs, int M, int nsm) {
  const int64_t rows = (nrs + kUpdRows - 1) / kUpdRows;
  const int64_t r = std::min<int64_t>(6 * (int64_t)nsm / rows, M / 64);
  return (int)std::max<int64_t>(1, r);
}

template <int NK>
static void launch_update_nk(const ChoUpd& u, cudaStream_t st) {
  if (u.nrange)
    k_cho_subtr<NK><<<dim3((unsigned)((u.nrs + kUpdRows - 1) / kUpdRows), u.nrange), kUpdThreads, 0, st>>>(u);
  k_cho_compvec<NK><<<(unsigned)((u.nrs + kUpdThreads - 1) / kUpdThreads), kUpdThreads, 0, st>>>(u);
  g_launches.fetch_add(u.nrange ? 2 : 1, std::memory_order_relaxed);
}
static void launch_update(ChoUpd u, int nsm, cudaStream_t st) {
  const int Mp = u.M + u.i0;
  const int want = Mp ? upd_ranges(u.nrs, Mp, nsm) : 0;
  u.jper = want ? ((Mp + want - 1) / want + kUpdJ - 1) / kUpdJ * kUpdJ : kUpdJ;
  u.nrange = (Mp + u.jper - 1) / u.jper;
  if (u.ni <= 2) launch_update_nk<2>(u, st);
  else if (u.ni <= 4) launch_update_nk<4>(u, st);
  else if (u.ni <= 6) launch_update_nk<6>(u, st);
  else if (u.ni <= 8) launch_update_nk<8>(u, st);
  else if (u.ni <= 12) launch_update_nk<12>(u, st);
  else if (u.ni <= 16) launch_update_nk<16>(u, st);
  else if (u.ni <= 24) launch_update_nk<24>(u, st);
  else launch_update_nk<32>(u, st);
}

__global__ void k_init_red(double* __restrict__ diag, unsigned char* __restrict__ inred, int64_t n, double scrmax) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n) return;
  if (diag[t] < scrmax) {
    diag[t] = 0.0;
    inred[t] = 0;
  } else {
    inred[t] = 1;
  }
}

// inv[a*n + b] = inv[b*n + a] = t for every rs pair t (filled with -1 first:
// AO pairs of shell pairs without rows keep it)
__global__ void k_rs_inverse(const int* __restrict__ rs_a, const int* __restrict__ rs_b, int64_t nrs, int n,
                             int* __restrict__ inv) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nrs) return;
  const int a = rs_a[t], b = rs_b[t];
  inv[(size_t)a * n + b] = (int)t;
  inv[(size_t)b * n + a] = (int)t;
}

static inline unsigned nblk(int64_t n, int b = 256) { return (unsigned)((n + b - 1) / b); }

// --------------------------------------------------------------- host side
struct ChoState {
  int64_t nrs = 0;
  std::vector<int> rs_a, rs_b, rs_sp;
  std::vector<int64_t> sp_first;
  std::vector<int> sp_count;
  std::vector<RsDev> rsd;       // host copy of d_rs while the state is built
  char* d_tab = nullptr;        // one allocation holding the tables below
  RsDev* d_rs = nullptr;
  int* d_rs_a = nullptr;        // AO indices of each rs entry (device)
  int* d_rs_b = nullptr;
  int64_t* d_sp_first = nullptr;
  int* d_sp_count = nullptr;
  double* d_diag = nullptr;     // working diagonal
  double* d_diag0 = nullptr;    // exact (ab|ab)
  unsigned char* d_inred = nullptr;
  int* d_inv = nullptr;         // rs index of every AO pair (n x n, -1: no row), J/K
  std::vector<double*> Lblk;    // FP64 vector blocks, nrs x kVecBlock each
  int M = 0;
  std::vector<int> piv, pass_of;
  int npass = 0;
  short* d_lexp = nullptr;      // row exponents of the square L_J (mixed J/K), M x lexp_ld
  int lexp_ld = 0;
};

// The vectors' storage of a state about to be replaced, for the next
// decomposition of the same list (which frees what it does not use).  FP64 J/K
// and mg_cho_copy_vectors return while their kernels and copies still read the
// vectors on the caller's stream, and the next decomposition may come on
// another one: the device finishes before the storage is written again.
void cho_recycle(Handle* h, ChoState* c) {
  if (!c) return;
  cudaDeviceSynchronize();
  h->cho_spare.swap(c->Lblk);
  h->cho_spare_bytes = sizeof(double) * (size_t)c->nrs * kVecBlock;
  cho_free(c);
}

void cho_free(ChoState* c) {
  if (!c) return;
  cudaFree(c->d_tab); cudaFree(c->d_lexp);
  for (auto p : c->Lblk) cudaFree(p);
  delete c;
}

// AO-pair list in reduced-set order (plf_cho_diag.F90:60-72 conventions):
// every shell pair (keep == nullptr) or the shell pairs with keep[sp] set
// (the others get sp_first = -1 and no rows).  Replaces a previous list.
static void make_rs(Handle* h, ChoState* c, const std::vector<char>* keep = nullptr) {
  c->rs_a.clear(); c->rs_b.clear(); c->rs_sp.clear(); c->sp_first.clear(); c->sp_count.clear(); c->rsd.clear();
  const int ns = h->sh.size();
  for (int i = 0; i < ns; ++i)
    for (int j = 0; j <= i; ++j) {
      const int sp = pair_id(i, j);
      if (keep && !(*keep)[sp]) {
        c->sp_first.push_back(-1);
        c->sp_count.push_back(0);
        continue;
      }
      const ShellH &A = h->sh[i], &B = h->sh[j];
      const int nA = A.nc * A.ncomp, nB = B.nc * B.ncomp;
      c->sp_first.push_back(c->rs_a.size());
      auto push = [&](int la, int lb) {
        c->rs_a.push_back(A.off + la);
        c->rs_b.push_back(B.off + lb);
        c->rs_sp.push_back(sp);
        RsDev r;
        r.sp = sp;
        r.ma = la / A.nc; r.ka = la % A.nc;
        r.mb = lb / B.nc; r.kb = lb % B.nc;
        c->rsd.push_back(r);
      };
      if (i != j) {
        for (int lb = 0; lb < nB; ++lb)
          for (int la = 0; la < nA; ++la) push(la, lb);
      } else {
        for (int la = 0; la < nA; ++la)
          for (int lb = 0; lb <= la; ++lb) push(la, lb);
      }
      c->sp_count.push_back((int)(c->rs_a.size() - c->sp_first.back()));
    }
  c->nrs = c->rs_a.size();
}

// The state's device tables, in one allocation; the rs list goes up in stream
// order.  The inverse table of the J/K calls is made here, too: the decomposition
// waits for its stream anyway, and FP64 J/K calls, the first one included, only queue.
static bool upload_rs(Handle* h, ChoState* c, cudaStream_t st) {
  const size_t n = std::max<int64_t>(c->nrs, 1), nsp = c->sp_first.size();
  size_t need = 0;
  auto place = [&](size_t bytes) { const size_t o = need; need += (bytes + 255) & ~(size_t)255; return o; };
  const size_t o_rs = place(sizeof(RsDev) * n), o_a = place(sizeof(int) * n), o_b = place(sizeof(int) * n),
               o_f = place(sizeof(int64_t) * nsp), o_c = place(sizeof(int) * nsp), o_d = place(sizeof(double) * n),
               o_d0 = place(sizeof(double) * n), o_in = place(n), o_inv = place(sizeof(int) * (size_t)h->nbf * h->nbf);
  if (dev_malloc(h, &c->d_tab, need) != cudaSuccess) return false;
  c->d_rs = (RsDev*)(c->d_tab + o_rs);
  c->d_rs_a = (int*)(c->d_tab + o_a);
  c->d_rs_b = (int*)(c->d_tab + o_b);
  c->d_sp_first = (int64_t*)(c->d_tab + o_f);
  c->d_sp_count = (int*)(c->d_tab + o_c);
  c->d_diag = (double*)(c->d_tab + o_d);
  c->d_diag0 = (double*)(c->d_tab + o_d0);
  c->d_inred = (unsigned char*)(c->d_tab + o_in);
  c->d_inv = (int*)(c->d_tab + o_inv);
  cudaMemcpyAsync(c->d_rs, c->rsd.data(), sizeof(RsDev) * c->nrs, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(c->d_rs_a, c->rs_a.data(), sizeof(int) * c->nrs, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(c->d_rs_b, c->rs_b.data(), sizeof(int) * c->nrs, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(c->d_sp_first, c->sp_first.data(), sizeof(int64_t) * nsp, cudaMemcpyHostToDevice, st);
  cudaMemcpyAsync(c->d_sp_count, c->sp_count.data(), sizeof(int) * nsp, cudaMemcpyHostToDevice, st);
  cudaMemsetAsync(c->d_inv, 0xFF, sizeof(int) * (size_t)h->nbf * h->nbf, st);
  k_rs_inverse<<<nblk(n), 256, 0, st>>>(c->d_rs_a, c->d_rs_b, c->nrs, h->nbf, c->d_inv);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  std::vector<RsDev>().swap(c->rsd);
  return true;
}

// ERI blocks (q4 quartets) into a scratch buffer; offsets per quartet
static double* eri_blocks(Handle* h, const std::vector<int32_t>& q4, std::vector<int64_t>& off, cudaStream_t st,
                          int& rc) {
  const int64_t nq = q4.size() / 4;
  off.assign(nq + 1, 0);
  for (int64_t t = 0; t < nq; ++t) {
    int64_t n = 1;
    for (int x = 0; x < 4; ++x) n *= (int64_t)h->sh[q4[4 * t + x]].nc * h->sh[q4[4 * t + x]].ncomp;
    off[t + 1] = off[t] + n;
  }
  const size_t need = sizeof(double) * std::max<int64_t>(off[nq], 1);
  double* buf = (double*)keep_get(h, h->cho_buf, need, st);
  if (!buf) { rc = MG_ERR_MEMORY; return nullptr; }
  std::vector<EriItem> items;
  std::vector<EriClass> classes;
  rc = build_eri_items(h, q4.data(), nq, off.data(), items, classes);
  if (rc) return nullptr;
  rc = run_eri_items(h, items, classes, buf, st);
  return buf;
}

static double cho_default_damp(double thrcom) {  // cho_setdamp.F90
  if (thrcom > 9.99e-3) return 1e7;
  if (thrcom > 9.99e-4) return 1e6;
  if (thrcom > 9.99e-5) return 1e5;
  if (thrcom > 9.99e-6) return 1e4;
  if (thrcom > 9.99e-7) return 1e3;
  if (thrcom > 9.99e-8) return 1e2;
  if (thrcom > 9.99e-9) return 1e1;
  return 1.0;
}

// CD_InCore_1p on the host (identical arithmetic to the reference)
static int cd_incore_1p(std::vector<double>& X, int n, std::vector<double>& Vec, int& numcho, double thr,
                        std::vector<int>& iD) {
  const double thrneg = -1e-13, thrfail = -1e-8;
  numcho = 0;
  const double acc = std::min(1e-12, thr * 1e-2);
  auto x = [&](int i, int j) -> double& { return X[i + (size_t)n * j]; };
  for (int pass = 0; pass < n; ++pass) {
    if (x(0, 0) < thrneg) {
      if (x(0, 0) < thrfail) return 101;
      for (int t = 0; t < n; ++t) { x(t, 0) = 0; x(0, t) = 0; }
    }
    double xmax = 0;
    int imax = -1;
    for (int i = 0; i < n; ++i) {
      if (x(i, i) < thrneg) {
        if (x(i, i) < thrfail) return 101;
        for (int t = 0; t < n; ++t) { x(t, i) = 0; x(i, t) = 0; }
      }
      if (x(i, i) > xmax + acc) { xmax = x(i, i); imax = i; }
    }
    if (xmax <= thr) return 0;
    const double xfac = 1.0 / std::sqrt(std::fabs(xmax));
    for (int j = 0; j < numcho; ++j) {
      const double v = Vec[imax + (size_t)n * j];
      for (int t = 0; t < n; ++t) x(t, imax) -= v * Vec[t + (size_t)n * j];
    }
    x(imax, imax) = xmax;
    const int k = numcho++;
    for (int i = 0; i < n; ++i) Vec[i + (size_t)n * k] = (x(i, i) == 0.0) ? 0.0 : xfac * x(i, imax);
    for (int i = 0; i < n; ++i) x(i, i) -= Vec[i + (size_t)n * k] * Vec[i + (size_t)n * k];
    x(imax, imax) = 0.0;
    iD.push_back(imax);
  }
  return 0;
}

// Static side of the per-pass integral batches: the kept shell pairs grouped by
// la + lb, heaviest (most primitive pairs) first, their block sizes and the
// distinct kinds of pair in each group, from which a pass's class statistics
// follow.  The ket of a pass is one shell pair, so nothing is sorted per pass.
struct ChoKind {
  int nij, ne, nsab, maxnp;
};
struct ChoItemPlan {
  std::vector<int> order[2 * MG_MAX_L + 1];       // shell pairs of la + lb = nab
  std::vector<ChoKind> kinds[2 * MG_MAX_L + 1];
  std::vector<int> kind_of;                        // per shell pair, in its group
  std::vector<int64_t> base;                       // first element of the bra block
  int64_t total = 0;                               // elements of all bra blocks
};

static void make_item_plan(const Handle* h, const ChoState* c, ChoItemPlan& p) {
  const int nsp = c->sp_count.size();
  p.kind_of.assign(nsp, 0);
  p.base.assign(nsp, 0);
  for (int sp = 0; sp < nsp; ++sp) {
    if (!c->sp_count[sp]) continue;
    const DPair& P = h->pairs[sp];
    const int nij = P.nci * P.ncj, nsab = P.nsa * P.nsb, nab = P.la + P.lb;
    p.base[sp] = p.total;
    p.total += (int64_t)nij * nsab;
    p.order[nab].push_back(sp);
    auto& ks = p.kinds[nab];
    size_t k = 0;
    while (k < ks.size() && !(ks[k].nij == nij && ks[k].ne == P.ne && ks[k].nsab == nsab)) ++k;
    if (k == ks.size()) ks.push_back({nij, P.ne, nsab, 0});
    ks[k].maxnp = std::max(ks[k].maxnp, P.np);
    p.kind_of[sp] = (int)k;
  }
  for (auto& o : p.order)
    std::stable_sort(o.begin(), o.end(), [&](int a, int b) { return h->pairs[a].np > h->pairs[b].np; });
}

// The (CD|AB) work items of one pass (bra pairs with alive[sp] != 0, ket spab)
static int pass_items(Handle* h, const ChoItemPlan& p, const unsigned char* alive, int spab,
                      std::vector<EriItem>& items, std::vector<EriClass>& classes) {
  const DPair& Q = h->pairs[spab];
  const int nkl = Q.nci * Q.ncj, ncd = Q.la + Q.lb;
  const int64_t ksz = (int64_t)nkl * Q.nsa * Q.nsb;
  items.clear();
  classes.clear();
  std::vector<char> seen;
  std::vector<int> chunk;
  for (int nab = 0; nab <= 2 * MG_MAX_L; ++nab) {
    if (p.order[nab].empty()) continue;
    const auto& ks = p.kinds[nab];
    seen.assign(ks.size(), 0);
    chunk.resize(ks.size());
    for (size_t k = 0; k < ks.size(); ++k) chunk[k] = eri_ket_chunk(ks[k].nij, ks[k].ne * Q.ne);
    EriClass c;
    c.nab = nab;
    c.ncd = ncd;
    c.begin = (int)items.size();
    c.work = 0;
    for (int sp : p.order[nab]) {
      if (!alive[sp]) continue;
      const int kd = p.kind_of[sp];
      if (chunk[kd] < 1) { h->err = "mg_cho_drv: bra contraction block too large"; return MG_ERR_ARG; }
      seen[kd] = 1;
      c.work += h->pairs[sp].np;
      for (int c0 = 0; c0 < nkl; c0 += chunk[kd])
        items.push_back({sp, spab, c0, std::min(nkl, c0 + chunk[kd]), (long long)(p.base[sp] * ksz)});
    }
    c.count = (int)items.size() - c.begin;
    if (!c.count) continue;
    ClassStats cs;
    for (size_t k = 0; k < ks.size(); ++k)
      if (seen[k]) eri_class_stats(cs, ks[k].nij, std::min(nkl, chunk[k]), ks[k].ne, Q.ne, ks[k].nsab, ks[k].maxnp, Q.np);
    c.work *= (double)Q.np * cs.max_nef;
    c.plan = eri_plan_for(h, nab, ncd, cs, c.count);
    if (c.plan.PAB < 1) { h->err = "mg_cho_drv: class does not fit in shared memory"; return MG_ERR_ARG; }
    classes.push_back(c);
  }
  return 0;
}

int cho_decompose(Handle* h, const ChoCfgH& cfg, ChoState*& out, cudaStream_t st, std::string& err) {
  ChoState* c = new ChoState;
  out = c;
  make_rs(h, c);
  const int nsp = c->sp_count.size();
  const double damp = cho_default_damp(cfg.thrcom);
  // the handle's buffers, kept for the next decomposition unless they are large
  struct Running {
    Handle* h;
    explicit Running(Handle* hh) : h(hh) { h->cho_running = true; }
    ~Running() {
      for (Workspace* w : {&h->cho_scr, &h->cho_buf, &h->cho_lq, &h->cho_upd})
        if (w->size > kKeepBytes) {
          cudaFree(w->ptr);
          *w = Workspace{};
        }
      give_back(h);  // the replaced vectors' storage that was not used
      h->cho_running = false;
    }
  } running(h);
  int rc = 0;
  // ---- diagonal (CHO_GETDIAG): (AB|AB) for every shell pair, then the initial
  // screening (cho_calcdiag.F90:255-300): elements below
  // ScrMax = ThrCom^2 / (Damp DiaMax) leave the reduced set.  The vectors are
  // stored over the shell pairs that keep at least one element (their rows
  // outside a pass's reduced set are zero), so the rs list is rebuilt over them.
  double scrmax = 1e15;
  {
    std::vector<int32_t> q4;
    for (int sp = 0; sp < nsp; ++sp) {
      const int i = h->pairs[sp].i, j = h->pairs[sp].j;
      q4.insert(q4.end(), {i, j, i, j});
    }
    std::vector<int64_t> off;
    double* buf = eri_blocks(h, q4, off, st, rc);
    if (rc) { err = "diagonal integrals failed: " + err; return rc; }
    // full diagonal, every shell pair
    const size_t rs_bytes = (sizeof(RsDev) * c->nrs + 255) & ~(size_t)255;
    char* d = (char*)keep_get(h, h->cho_scr, rs_bytes + sizeof(int64_t) * nsp + sizeof(double) * c->nrs, st);
    if (!d) { err = "diagonal: out of device memory"; return MG_ERR_MEMORY; }
    RsDev* d_rs = (RsDev*)d;
    int64_t* d_off = (int64_t*)(d + rs_bytes);
    double* d_full = (double*)(d_off + nsp);
    cudaMemcpyAsync(d_rs, c->rsd.data(), sizeof(RsDev) * c->nrs, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(d_off, off.data(), sizeof(int64_t) * nsp, cudaMemcpyHostToDevice, st);
    k_extract_diag<<<nblk(c->nrs), 256, 0, st>>>(d_rs, c->nrs, h->d_pairs, d_off, buf, d_full);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    std::vector<double> hd(c->nrs);
    cudaMemcpyAsync(hd.data(), d_full, sizeof(double) * c->nrs, cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    double dm = 0;
    for (double v : hd) dm = std::max(dm, std::fabs(v));
    if (dm > 0) scrmax = cfg.thrcom * cfg.thrcom / damp / dm;
    std::vector<char> keep(nsp, 0);
    for (int64_t t = 0; t < c->nrs; ++t)
      if (!(hd[t] < scrmax)) keep[c->rs_sp[t]] = 1;
    make_rs(h, c, &keep);
    // the diagonal over the kept shell pairs, from the same integral blocks
    if (!upload_rs(h, c, st)) { err = "diagonal: out of device memory"; return MG_ERR_MEMORY; }
    k_extract_diag<<<nblk(std::max<int64_t>(c->nrs, 1)), 256, 0, st>>>(c->d_rs, c->nrs, h->d_pairs, d_off, buf,
                                                                        c->d_diag0);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    cudaMemcpyAsync(c->d_diag, c->d_diag0, sizeof(double) * c->nrs, cudaMemcpyDeviceToDevice, st);
    cudaStreamSynchronize(st);
  }
  const int64_t nrs = c->nrs;
  const size_t blk_bytes = sizeof(double) * (size_t)nrs * kVecBlock;
  if (h->cho_spare_bytes != blk_bytes) give_back(h);  // the previous vectors' storage fits the same list only
  ChoItemPlan plan;
  make_item_plan(h, c, plan);
  int maxcnt = 1;
  for (int sp = 0; sp < nsp; ++sp) maxcnt = std::max(maxcnt, c->sp_count[sp]);
  const int MQ = std::min(cfg.maxqual, maxcnt);  // the qualified columns belong to one shell pair
  const int maxblk = cfg.maxvec / kVecBlock + 2;
  // CTAs of k_cho_lq (each holds a partial qualified block), at most 64 MB of them
  const int kParts = (int)std::max<int64_t>(1, std::min<int64_t>(148, ((int64_t)8 << 20) / ((int64_t)MQ * MQ)));
  if (!smem_attr_once((const void*)k_cho_lq, 200 * 1024)) { err = "shared-memory limit could not be raised"; return MG_ERR_CUDA; }
  // ---- scratch of the passes, one allocation
  size_t need = 0;
  auto place = [&](size_t bytes) { const size_t o = need; need += (bytes + 255) & ~(size_t)255; return o; };
  const size_t sel_bytes = sizeof(ChoSel) + sizeof(double) * maxcnt + (size_t)(maxcnt + 7) / 8 * 8 + nsp;
  const size_t par_bytes = sizeof(double) * ((size_t)MQ + (size_t)MQ * MQ) + sizeof(int) * 2 * MQ;
  const size_t o_sel = place(sel_bytes), o_diash = place(sizeof(double) * 2 * nsp), o_par = place(par_bytes),
               o_base = place(sizeof(int64_t) * nsp), o_lt = place(sizeof(double*) * maxblk), o_xm = place(16),
               o_cols = place(sizeof(int) * MQ), o_q = place(sizeof(double) * MQ * MQ),
               o_part = place(sizeof(double) * MQ * MQ * kParts);
  char* scr = (char*)keep_get(h, h->cho_scr, need, st);
  // partial sums of the update kernels
  const int nrow = (int)((nrs + kUpdRows - 1) / kUpdRows);
  const size_t upd = sizeof(double) * std::max<size_t>(1, 6 * h->nsm / std::max(nrow, 1)) * std::min(32, MQ) * std::max<int64_t>(nrs, 1);
  double* d_upd = (double*)keep_get(h, h->cho_upd, upd, st);
  if (!scr || !d_upd) { err = "out of device memory for the passes' scratch"; return MG_ERR_MEMORY; }
  ChoSel* d_sel = (ChoSel*)(scr + o_sel);
  double* d_dpair = (double*)(d_sel + 1);
  unsigned char* d_rpair = (unsigned char*)(d_dpair + maxcnt);
  unsigned char* d_alive = d_rpair + (size_t)(maxcnt + 7) / 8 * 8;
  double* d_diash = (double*)(scr + o_diash);
  double* d_par = (double*)(scr + o_par);
  int64_t* d_base = (int64_t*)(scr + o_base);
  double** d_lt = (double**)(scr + o_lt);
  unsigned long long* d_xm = (unsigned long long*)(scr + o_xm);
  int* d_flags = (int*)(d_xm + 1);
  int* d_cols = (int*)(scr + o_cols);
  double* d_Q = (double*)(scr + o_q);
  double* d_part = (double*)(scr + o_part);
  // host side of the same, pinned: the select buffer, Q, the parameters
  const size_t pin_sel = (sel_bytes + 255) & ~(size_t)255, pin_q = sizeof(double) * MQ * MQ;
  char* pin = (char*)pin_get(h, pin_sel + ((pin_q + 255) & ~(size_t)255) + par_bytes);
  if (!pin) { err = "pinned host memory for the passes"; return MG_ERR_MEMORY; }
  const ChoSel* hsel = (const ChoSel*)pin;
  const double* hdpair = (const double*)(hsel + 1);
  const unsigned char* hrpair = (const unsigned char*)(hdpair + maxcnt);
  const unsigned char* halive = hrpair + (size_t)(maxcnt + 7) / 8 * 8;
  double* hQ = (double*)(pin + pin_sel);
  double* hpar = (double*)(pin + pin_sel + ((pin_q + 255) & ~(size_t)255));
  k_init_red<<<nblk(std::max<int64_t>(nrs, 1)), 256, 0, st>>>(c->d_diag, c->d_inred, nrs, scrmax);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  cudaMemsetAsync(d_xm, 0, 16, st);
  cudaMemcpyAsync(d_base, plan.base.data(), sizeof(int64_t) * nsp, cudaMemcpyHostToDevice, st);
  std::vector<EriItem> items;
  std::vector<EriClass> classes;
  std::vector<double> Q, Vec;
  std::vector<int> iD;
  for (int pass = 0; pass <= nrs; ++pass) {
    // ---- Cho_SetRed of the previous pass, Cho_SetPass and Cho_GetMaxShl; the
    // diagonal and the reduced-set flags of the chosen shell pair come along
    k_cho_scan<<<(nsp + 7) / 8, 256, 0, st>>>(c->d_diag, c->d_inred, c->d_sp_first, c->d_sp_count, nsp, d_xm, pass > 0,
                                              damp, cfg.thrcom, d_diash, d_alive);
    k_cho_select<<<1, 1024, 0, st>>>(d_diash, nsp, cfg.thrcom, c->d_sp_first, c->d_sp_count, c->d_diag, c->d_inred,
                                     d_flags, d_xm, d_sel, d_dpair, d_rpair);
    g_launches.fetch_add(2, std::memory_order_relaxed);
    cudaMemcpyAsync(pin, d_sel, sel_bytes, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) { rc = MG_ERR_CUDA; err = "CUDA error in Cholesky pass"; break; }
    if (hsel->flags) { rc = MG_ERR_DECOMP; err = "diagonal too negative (Cho_ChkDia_A4 TooNeg)"; break; }
    const double dgmax = hsel->dgmax;  // max |diagonal| over the reduced set
    if (dgmax < cfg.thrcom) break;
    const double diamin = std::max(dgmax * cfg.span, cfg.thrcom);
    const double smax = hsel->smax;
    const int spab = hsel->spab;
    if (smax == 0.0 || std::fabs(smax) < diamin) { rc = MG_ERR_DECOMP; err = "no qualifying diagonal (Cho_GetInt 104)"; break; }
    // ---- Cho_Qualify_2 within shell pair spab (cho_qualify.h): positions t
    // inside the pair, then rs indices
    std::vector<int> qual = cho_qualify_2(hdpair, hrpair, c->sp_count[spab], diamin, cfg.maxqual);
    for (int& t : qual) t = (int)(c->sp_first[spab] + t);
    const int nq = qual.size();
    if (nq == 0) { rc = MG_ERR_DECOMP; err = "empty qualification (Cho_GetInt 104)"; break; }
    // ---- integral columns (CD|AB) for every CD pair touching the reduced set
    const DPair& A = h->pairs[spab];
    const int64_t ksz = (int64_t)A.nci * A.ncj * A.nsa * A.nsb;
    double* buf = (double*)keep_get(h, h->cho_buf, sizeof(double) * std::max<int64_t>(plan.total * ksz, 1), st);
    if (!buf) { rc = MG_ERR_MEMORY; err = "column integrals failed: out of device memory"; break; }
    rc = pass_items(h, plan, halive, spab, items, classes);
    if (!rc) rc = run_eri_items(h, items, classes, buf, st);
    if (rc) { err = "column integrals failed: " + err; break; }
    // ---- Cho_Dec_Qual: Q = MQ - LQ LQ^T  (MQ: the columns' rows at the qualified positions)
    const int M = c->M;
    double* d_lq = (double*)h->cho_lq.ptr;
    if (h->cho_lq.size < sizeof(double) * (size_t)nq * (M + nq)) {  // grows with the vectors
      d_lq = (double*)keep_get(h, h->cho_lq, sizeof(double) * (size_t)MQ * (M + kVecBlock + MQ), st);
      if (!d_lq) { rc = MG_ERR_MEMORY; err = "out of device memory for the LQ rows"; break; }
    }
    cudaMemcpyAsync(d_cols, qual.data(), sizeof(int) * nq, cudaMemcpyHostToDevice, st);
    int nparts = 0;
    if (M > 0) {
      const int jb = std::max(1, std::min(64, 6144 / nq));
      nparts = std::min((M + jb - 1) / jb, kParts);
      k_cho_lq<<<nparts, 256, sizeof(double) * jb * nq, st>>>(d_lt, nrs, M, d_cols, nq, jb, d_lq, d_part);
      g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    k_cho_q<<<nblk((int64_t)nq * nq, 128), 128, 0, st>>>(c->d_rs, h->d_pairs, buf + plan.base[spab] * ksz, d_cols, nq,
                                                         spab, d_part, nparts, d_Q);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    cudaMemcpyAsync(hQ, d_Q, sizeof(double) * nq * nq, cudaMemcpyDeviceToHost, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) { rc = MG_ERR_CUDA; err = "CUDA error in Cholesky pass"; break; }
    Q.assign(hQ, hQ + (size_t)nq * nq);
    // Cho_P_MaxDX is the largest diagonal of the reduced set, all of them positive: dgmax
    const double thr = std::max(cfg.thrcom, dgmax * cfg.span);
    Vec.assign((size_t)nq * nq, 0.0);
    iD.clear();
    int nk = 0;
    if (cd_incore_1p(Q, nq, Vec, nk, thr, iD)) { rc = MG_ERR_DECOMP; err = "CD_InCore_1p failed (negative diagonal)"; break; }
    if (nk == 0) { rc = MG_ERR_DECOMP; err = "no vector from qualified block"; break; }
    if (M + nk > cfg.maxvec) { rc = MG_ERR_MEMORY; err = "too many Cholesky vectors (MaxVec)"; break; }
    // pivot order (cho_decom_a4.F90:120-170)
    double *fac = hpar, *K = hpar + nk;
    int *qrs = (int*)(K + (size_t)nk * nk), *colsel = qrs + nk;
    std::vector<double> qd(nk);
    for (int i = 0; i < nk; ++i)
      for (int j = 0; j < nk; ++j) K[j + (size_t)nk * i] = Vec[iD[j] + (size_t)nq * i];
    for (int i = 0; i < nk; ++i) { qd[i] = hQ[iD[i] + (size_t)nq * iD[i]]; qrs[i] = qual[iD[i]]; colsel[i] = iD[i]; }
    const double qdmax = qd[0];
    for (int i = 0; i < nk; ++i) {
      fac[i] = 1.0 / std::sqrt(std::fabs(qd[i]));
      for (int j = i; j < nk; ++j) qd[j] -= K[j + (size_t)nk * i] * K[j + (size_t)nk * i];
      qd[i] = 0.0;
    }
    // storage of this pass's vectors (every element of a column is written)
    while ((int)c->Lblk.size() * kVecBlock < M + nk) {
      double* p = nullptr;
      if (!h->cho_spare.empty()) {
        p = h->cho_spare.back();
        h->cho_spare.pop_back();
      } else if (dev_malloc(h, &p, blk_bytes) != cudaSuccess) {
        rc = MG_ERR_MEMORY;
        break;
      }
      cudaMemcpyAsync(d_lt + c->Lblk.size(), &p, sizeof(double*), cudaMemcpyHostToDevice, st);
      c->Lblk.push_back(p);
    }
    if (rc) { err = "out of device memory for Cholesky vectors"; break; }
    cudaMemcpyAsync(d_par, hpar, sizeof(double) * ((size_t)nk + (size_t)nk * nk) + sizeof(int) * 2 * nk,
                    cudaMemcpyHostToDevice, st);
    if (nk > 32)  // later launches read the LQ rows of this pass's own vectors
      cudaMemcpyAsync(d_lq + (size_t)M * nq, Vec.data(), sizeof(double) * (size_t)nq * nk, cudaMemcpyHostToDevice, st);
    // ---- Cho_Subtr and Cho_CompVec
    ChoUpd u{d_lt, nrs, M, 0, 0, nk, nq, spab, 0, 0, 0, d_upd, d_lq, buf, d_base, ksz, c->d_rs, h->d_pairs, c->d_inred, c->d_diag,
             d_par, (const int*)(d_par + nk + (size_t)nk * nk), qdmax, damp, cfg.thrcom, -1e-40, -1e-8, d_flags, d_xm};
    for (u.i0 = 0; u.i0 < nk; u.i0 += 32) {
      u.ni = std::min(32, nk - u.i0);
      u.last = u.i0 + 32 >= nk;
      launch_update(u, h->nsm, st);
    }
    for (int i = 0; i < nk; ++i) { c->piv.push_back(qrs[i]); c->pass_of.push_back(pass); }
    c->M = M + nk;
    c->npass = pass + 1;
    if (cudaGetLastError() != cudaSuccess) { rc = MG_ERR_CUDA; err = "CUDA error in Cholesky pass"; break; }
  }
  cudaStreamSynchronize(st);
  return rc;
}

int64_t cho_nrs(const ChoState* c) { return c->nrs; }
int cho_nvec(const ChoState* c) { return c->M; }
int cho_npass(const ChoState* c) { return c->npass; }
void cho_pivots(const ChoState* c, int32_t* piv, int32_t* pass_of) {
  for (int k = 0; k < c->M; ++k) {
    if (piv) piv[k] = c->piv[k];
    if (pass_of) pass_of[k] = c->pass_of[k];
  }
}
void cho_rs_list(const ChoState* c, int32_t* a, int32_t* b, int32_t* sp) {
  for (int64_t t = 0; t < c->nrs; ++t) {
    if (a) a[t] = c->rs_a[t];
    if (b) b[t] = c->rs_b[t];
    if (sp) sp[t] = c->rs_sp[t];
  }
}
int cho_copy_vectors(const ChoState* c, int first, int count, double* d_out, cudaStream_t st) {
  if (first < 0 || count < 0 || first + count > c->M) return MG_ERR_ARG;
  for (int k = 0; k < count;) {  // one copy per storage block
    const int J = first + k, n = std::min(count - k, kVecBlock - J % kVecBlock);
    cudaMemcpyAsync(d_out + c->nrs * k, c->Lblk[J / kVecBlock] + (size_t)c->nrs * (J % kVecBlock),
                    sizeof(double) * c->nrs * n, cudaMemcpyDeviceToDevice, st);
    k += n;
  }
  return 0;
}
const double* cho_diag0(const ChoState* c) { return c->d_diag0; }
const int* cho_rs_a_dev(const ChoState* c) { return c->d_rs_a; }
const int* cho_rs_b_dev(const ChoState* c) { return c->d_rs_b; }
// contiguous FP64 vectors [J0, J0+nb) (the range must not cross a storage block)
const double* cho_vec_ptr(const ChoState* c, int J0, int nb, cudaStream_t, Handle*) {
  if (J0 / kVecBlock != (J0 + nb - 1) / kVecBlock) return nullptr;
  return c->Lblk[J0 / kVecBlock] + (size_t)c->nrs * (J0 % kVecBlock);
}
int cho_vec_block() { return kVecBlock; }
short* cho_lexp(const ChoState* c, int ld) { return c->lexp_ld == ld ? c->d_lexp : nullptr; }
void cho_set_lexp(ChoState* c, short* p, int ld) {
  cudaFree(c->d_lexp);
  c->d_lexp = p;
  c->lexp_ld = ld;
}

const int* cho_inv_dev(const ChoState* c) { return c->d_inv; }

// ------------------------------------------------- in-core decomposition
// CD_InCore (cholesky_util/cd_incore.F90:14 -> cd_incore_1.F90): pivoted
// Cholesky factor of a symmetric positive semidefinite n x n matrix X, left
// looking: each step takes the largest remaining diagonal (the first one,
// in index order, that exceeds the running maximum by more than
// Acc = min(1e-12, Thr/100)), updates only the pivot column against the
// previous vectors, scales it into the new vector and subtracts its square
// from the diagonal; diagonals below ThrNeg = -1e-13 are zeroed with their
// row and column, below ThrFail = -1e-8 the decomposition fails (irc 101);
// it stops when the largest diagonal is <= Thr.  One CTA, bound by the latency
// of one step (some ten barriers and two rounds of loads).  The pivot: the
// block's maximum and its first index; the running-maximum rule gives that
// element whenever no other diagonal lies within 2 Acc of it, otherwise thread 0
// scans in index order.  The pivot's row of the vectors is staged in shared
// memory; the column update, the new vector and the diagonal update are
// row-parallel.  41 vectors of a 300 x 300 density: 683 us with a serial scan and
// a serial chain of loads per row, 119 us this way.
// out[0] = NumCho, out[1] = irc (0, 101, 102).
constexpr int kCdThreads = 1024;
constexpr int kCdStaged = 10000;  // largest n whose pivot row fits in shared memory beside the rest

__global__ void __launch_bounds__(kCdThreads) k_cd_incore(double* __restrict__ X, int n, double* __restrict__ Vec,
                                                          int maxvec, double thr, int* __restrict__ out) {
  // the diagonal of X, the pivot's row of Vec (up to kCdStaged), then n ints of zeroed indices
  extern __shared__ double cd_dg[];
  double* prow = cd_dg + n;
  const bool staged = n <= kCdStaged;
  int* zl = reinterpret_cast<int*>(staged ? prow + n : prow);
  __shared__ double sg[kCdThreads / 32];
  __shared__ int si[kCdThreads / 32];
  __shared__ int s_imax, s_nz, s_near;
  __shared__ double s_xmax;
  const double thrneg = -1.0e-13, thrfail = -1.0e-8;
  const double acc = fmin(1.0e-12, thr * 1.0e-2);
  const int tid = threadIdx.x, lane = tid & 31;
  for (int i = tid; i < n; i += blockDim.x) cd_dg[i] = X[i + (size_t)n * i];
  if (tid == 0) s_nz = s_near = 0;
  __syncthreads();
  int numcho = 0, irc = 0;
  for (int pass = 0; pass < n; ++pass) {
    double g = -1.0;
    int idx = 0x7fffffff;
    bool fail = false;
    for (int i = tid; i < n; i += blockDim.x) {
      double d = cd_dg[i];
      if (d < thrneg) {
        if (d < thrfail) fail = true;
        d = 0.0;
        cd_dg[i] = 0.0;
        zl[atomicAdd(&s_nz, 1)] = i;
      }
      if (d > g) { g = d; idx = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double g2 = __shfl_xor_sync(0xffffffffu, g, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
      if (g2 > g || (g2 == g && i2 < idx)) { g = g2; idx = i2; }
    }
    if (lane == 0) { sg[tid >> 5] = g; si[tid >> 5] = idx; }
    if (__syncthreads_or(fail)) { irc = 101; break; }
    g = sg[lane];
    idx = si[lane];
    for (int o = 16; o > 0; o >>= 1) {
      const double g2 = __shfl_xor_sync(0xffffffffu, g, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
      if (g2 > g || (g2 == g && i2 < idx)) { g = g2; idx = i2; }
    }
    int near = 0;  // diagonals the running-maximum rule could prefer
    for (int i = tid; i < n; i += blockDim.x) near += cd_dg[i] > g - 2.0 * acc;
    if (near) atomicAdd(&s_near, near);
    __syncthreads();
    int imax = idx;
    double xmax = g > acc ? g : 0.0;
    if (s_near != 1) {
      if (tid == 0) {
        imax = -1;
        xmax = 0.0;
        for (int i = 0; i < n; ++i)
          if (cd_dg[i] > xmax + acc) {
            xmax = cd_dg[i];
            imax = i;
          }
        s_imax = imax;
        s_xmax = xmax;
      }
      __syncthreads();
      imax = s_imax;
      xmax = s_xmax;
    }
    if (!(xmax > thr)) break;  // converged
    if (numcho == maxvec) { irc = 102; break; }
    if (staged)
      for (int j = tid; j < numcho; j += blockDim.x) prow[j] = Vec[imax + (size_t)n * j];
    for (int z = 0; z < s_nz; ++z) {  // rows and columns of the zeroed diagonals
      const int iz = zl[z];
      for (int k = tid; k < n; k += blockDim.x) {
        X[k + (size_t)n * iz] = 0.0;
        X[iz + (size_t)n * k] = 0.0;
      }
    }
    __syncthreads();
    const double xfac = 1.0 / sqrt(fabs(xmax));
    double* vnew = Vec + (size_t)n * numcho;
    for (int i = tid; i < n; i += blockDim.x) {
      double x = X[i + (size_t)n * imax];
      const double* v = Vec + i;
      int j = 0;
      for (; staged && j + 8 <= numcho; j += 8) {
        double w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = v[(size_t)n * (j + e)];
#pragma unroll
        for (int e = 0; e < 8; ++e) x -= prow[j + e] * w[e];
      }
      for (; j < numcho; ++j) x -= (staged ? prow[j] : Vec[imax + (size_t)n * j]) * v[(size_t)n * j];
      if (i == imax) x = xmax;
      X[i + (size_t)n * imax] = x;
      const double vn = cd_dg[i] == 0.0 ? 0.0 : xfac * x;
      vnew[i] = vn;
      cd_dg[i] = i == imax ? 0.0 : cd_dg[i] - vn * vn;
    }
    if (tid == 0) s_nz = s_near = 0;
    ++numcho;
    __syncthreads();
  }
  if (tid == 0) {
    out[0] = numcho;
    out[1] = irc;
  }
}

int cd_incore(Handle* h, double* d_X, int n, double thr, double* d_vec, int maxvec, int* numcho, cudaStream_t st) {
  *numcho = 0;
  if (n < 1) return 0;
  if (maxvec < 1) return -1;
  if (thr < 0.0) thr = 1.0e-6;  // CD_InCore's DefThr
  const size_t smem = (size_t)n * ((n <= kCdStaged ? 2 : 1) * sizeof(double) + sizeof(int));
  if (smem > 200 * 1024) {
    h->err = "in-core decomposition: n above 17066";
    return MG_ERR_ARG;
  }
  if (!smem_attr_once((const void*)k_cd_incore, 200 * 1024)) {
    h->err = "in-core decomposition: shared-memory limit could not be raised";
    return MG_ERR_CUDA;
  }
  int* d_out = (int*)ws_get(h, 2 * sizeof(int), st);
  if (!d_out) { h->err = "workspace allocation failed"; return MG_ERR_MEMORY; }
  k_cd_incore<<<1, kCdThreads, smem, st>>>(d_X, n, d_vec, maxvec, thr, d_out);
  g_launches.fetch_add(1, std::memory_order_relaxed);
  int hout[2] = {0, 0};
  cudaMemcpyAsync(hout, d_out, sizeof(hout), cudaMemcpyDeviceToHost, st);
  if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    h->err = "in-core decomposition: CUDA error";
    return MG_ERR_CUDA;
  }
  *numcho = hout[0];
  return hout[1];
}

}  // namespace mg
