// Two-electron gradient kernel (FP64), one template instantiated per
// (la+lb+1, lc+ld+1) class; MINB (resident CTAs per SM) sets the threads per
// CTA and the register budget.  The algorithm and its reference anchors are
// described in grad.cu; the instantiations live in grad_k1.cu .. grad_k3.cu.
#pragma once
#include <cuda_runtime.h>

#include "kern_common.cuh"

namespace mg {

// Per-CTA table block (doubles), copied from global memory at kernel start:
// Cartesian -> spherical matrices for l = 0..3 (column m, row Cartesian) and
// the Cartesian exponents of l = 0..7 in C3 order packed as
// x | y << 8 | z << 16 (ints).
constexpr int kGTabSph = 0;
constexpr int kGTabCart = 110;  // 120 ints = 60 doubles
constexpr int kGTabD = 170;

struct GradArgs {
  const GradItem* items;
  int nitems;
  const DPair* pairs;
  const double* prim;
  int tot_np;
  const double* coef;
  const double* Dm;
  int nbf;
  const double* gtab;
  double* grad;
  double* scratch;       // per-group global slots: contracted 2-PDM + stage-0 temp
  long long scr_stride;  // doubles per slot
  int* counter;          // work-item counter of this launch (starts at 0)
  int tpq, gsm, PAB, PCD, RW;
  // 2-PDM of PGet1 (integral_util/pget1.F90:66-106):
  //   G = cq D(ab) D(cd) - xq [D(ac) D(bd) + D(ad) D(bc) + Ds(ac) Ds(bd) + Ds(ad) Ds(bc)]
  const double* Ds;  // spin density (open shell) or null
  double cq;         // CoulFac
  double xq;         // ExFac / 4
};

using GradFn = void (*)(GradArgs, RysArgs);
// the kernel of class (nab1, ncd1): instantiated in grad_k1.cu (nab1 1..3),
// grad_k2.cu (4, 5) and grad_k3.cu (6, 7), which compile side by side
GradFn grad_kernel_m1(int nab1, int ncd1);
GradFn grad_kernel_lo(int nab1, int ncd1);
GradFn grad_kernel_mid(int nab1, int ncd1);
GradFn grad_kernel_hi(int nab1, int ncd1);

// Assg1 for one shell quartet class whose fastest component indices run over
// shells of LA and LB (LB = 0: one shell), sum-factorised over the directions.
// With G the primitive density and X, Y, Z the 2D integrals of a component,
//   U[x] = sum G Y Z,  V[y] = sum G X Z,  W[z] = sum G X Y
// over the components that share the 2D index x (y, z), and a derivative
// factor multiplies U, V or W once per 2D index instead of once per component:
// five FP64 operations per component and root and nine per 2D index and
// direction, against fourteen per component for the products one by one, and the
// derivative factors (three of the four values of a record) are read once per 2D
// index.  A thread takes all NCA x NCB components of one (quartet, rest) and
// loops over the roots.  abcd0, the first component, is (LA, 0, 0) x (LB, 0, 0),
// so its packed x index lies LA + (LA + 1) LB after the block's first.
template <int LA, int LB>
__device__ __forceinline__ void assg1_block(const double* __restrict__ F, const double* __restrict__ Gp,
                                            const int* __restrict__ IX, int nt, int nrest, int St, int Gs, int J4,
                                            int nrw, int tid, int tpq, double* acc) {
  constexpr int NCA = (LA + 1) * (LA + 2) / 2, NCB = (LB + 1) * (LB + 2) / 2;
  constexpr int N = (LA + 1) * (LB + 1);  // 2D indices per direction
  constexpr CartExp<LA> ca{};
  constexpr CartExp<LB> cb{};
  const FDiv fnt = fdiv(nt);
  for (int w = tid; w < nt * nrest; w += tpq) {
    const int rest = fq(w, fnt), t = w - rest * nt;
    const int abcd0 = NCA * NCB * rest;
    const double* g = Gp + t * Gs + abcd0;
    const int pk = IX[abcd0];
    const double* Fx = F + (size_t)t * St + 4 * ((pk & 255) - (LA + (LA + 1) * LB));
    const double* Fy = F + (size_t)t * St + J4 + 4 * ((pk >> 8) & 255);
    const double* Fz = F + (size_t)t * St + 2 * J4 + 4 * (pk >> 16);
    constexpr bool kHold = NCA * NCB <= 6;  // the densities stay in registers over the roots
    double gh[kHold ? NCA * NCB : 1];
    if (kHold) {
#pragma unroll
      for (int c = 0; c < NCA * NCB; ++c) gh[kHold ? c : 0] = g[c];
    }
    for (int rl = 0; rl < nrw; ++rl, Fx += 3 * J4, Fy += 3 * J4, Fz += 3 * J4) {
      double X[N], Y[N], Z[N], U[N], V[N], W[N];
#pragma unroll
      for (int i = 0; i < N; ++i) {
        X[i] = Fx[4 * i];
        Y[i] = Fy[4 * i];
        Z[i] = Fz[4 * i];
        U[i] = V[i] = W[i] = 0.0;
      }
#pragma unroll
      for (int jb = 0; jb < NCB; ++jb)
#pragma unroll
        for (int ja = 0; ja < NCA; ++ja) {
          const int x = ca.e[ja][0] + (LA + 1) * cb.e[jb][0], y = ca.e[ja][1] + (LA + 1) * cb.e[jb][1],
                    z = ca.e[ja][2] + (LA + 1) * cb.e[jb][2];
          const double gm = kHold ? gh[kHold ? ja + NCA * jb : 0] : g[ja + NCA * jb];
          const double gx = gm * X[x], gy = gm * Y[y];
          U[x] = fma(gy, Z[z], U[x]);
          V[y] = fma(gx, Z[z], V[y]);
          W[z] = fma(gx, Y[y], W[z]);
        }
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const double2 dx = *reinterpret_cast<const double2*>(Fx + 4 * i + 2);
        const double2 dy = *reinterpret_cast<const double2*>(Fy + 4 * i + 2);
        const double2 dz = *reinterpret_cast<const double2*>(Fz + 4 * i + 2);
        acc[0] = fma(U[i], Fx[4 * i + 1], acc[0]);
        acc[1] = fma(V[i], Fy[4 * i + 1], acc[1]);
        acc[2] = fma(W[i], Fz[4 * i + 1], acc[2]);
        acc[3] = fma(U[i], dx.x, acc[3]);
        acc[4] = fma(V[i], dy.x, acc[4]);
        acc[5] = fma(W[i], dz.x, acc[5]);
        acc[6] = fma(U[i], dx.y, acc[6]);
        acc[7] = fma(V[i], dy.y, acc[7]);
        acc[8] = fma(W[i], dz.y, acc[8]);
      }
    }
  }
}

// s += c[0..3] v; AL: c is 16-byte aligned (two loads instead of four)
template <bool AL>
__device__ __forceinline__ void axpy4(const double* __restrict__ c, double v, double (&s)[4]) {
  double2 a, b;
  if (AL) {
    a = *reinterpret_cast<const double2*>(c);
    b = *reinterpret_cast<const double2*>(c + 2);
  } else {
    a = make_double2(c[0], c[1]);
    b = make_double2(c[2], c[3]);
  }
  s[0] = fma(a.x, v, s[0]);
  s[1] = fma(a.y, v, s[1]);
  s[2] = fma(b.x, v, s[2]);
  s[3] = fma(b.y, v, s[3]);
}

// Largest NI * NJ whose recursion stage runs one thread per job with the whole
// 2D table of the job (NI NJ doubles) and the transfer rows in registers.  Larger
// classes (from (3, 4): the registers spill more and more, and their tiles have
// too few jobs to hide one long thread) go through a table in shared memory.
// 460-function gradient, all classes with unchanged tiles 1723 -> 1554 ms: (3, 3)
// 167 -> 139, (2, 3) 78 -> 50, (2, 2) 28 -> 17; (3, 5) 103 -> 92, (4, 5) 120 -> 106,
// (5, 4) 110 -> 101.  The largest classes below the limit spill, too (bytes stored:
// (5, 2) 224, (4, 2) 176, (3, 3) 88, (2, 5) 68), and are the faster this way all
// the same: against the shared-memory table, each with its best tile, 10 atoms of
// 4s3p2d: (4, 2) 4.03 and 4.29 ms, (3, 3) 10.0 and 11.5, (2, 5) 2.63 and 2.71, the
// smaller tables 1.3 to 1.5 times as fast.  (5, 2) alone is slower, 3.05 and 3.00 (5
// atoms with f shells: 2.43 and 2.27), too little for a rule of its own.
constexpr int kGradJobMax = 18;

// The recursion stage with one thread per (quartet, root, direction) job.  The
// lane-per-row form (one NI-lane segment per job, rows exchanged by shuffles)
// spends NI lanes on values that one thread forms in as many instructions, and
// only la + 1 of the lanes store; a thread per job needs about a fifth of the
// instructions.  When a wave has fewer jobs than half the group's threads, up to
// four threads share a job: each repeats the recursion and takes every nsub-th
// (c, d) column.  A job record's stride is 2 mod 4 doubles, so the 16-byte
// stores of consecutive threads fall in different banks.
template <int NI, int NJ, int NR>
__device__ __forceinline__ void grad_jobs_thread(const double* __restrict__ cf, int CFT, const double* __restrict__ hdr,
                                                 double* __restrict__ F, int nt, int nrw, int r0, int la, int lb,
                                                 int lc, int ld, int J4, int St, const FDiv& fnrw, int tid, int tpq) {
  const int njobs = nt * nrw * 3;
  const int nsub = 4 * njobs <= tpq ? 4 : 2 * njobs <= tpq ? 2 : 1;
  for (int q = tid; q < njobs * nsub; q += tpq) {
    const int sub = q >= njobs ? (q >= 2 * njobs ? (q >= 3 * njobs ? 3 : 2) : 1) : 0, job = q - sub * njobs;
    const int tr = job / 3, d = job - 3 * tr, t = fq(tr, fnrw), rl = tr - t * nrw, r = r0 + rl;
    const double* c = cf + t * CFT + r * 10;
    const double B00 = c[0], B10 = c[1], B01 = c[2], C00 = c[3 + d], D00 = c[6 + d];
    double G[NJ][NI];  // G[j][e]
    G[0][0] = d == 2 ? c[9] : 1.0;
    G[0][1] = C00 * G[0][0];
#pragma unroll
    for (int i = 1; i < NI - 1; ++i) G[0][i + 1] = fma(i * B10, G[0][i - 1], C00 * G[0][i]);
#pragma unroll
    for (int j = 0; j < NJ - 1; ++j)
#pragma unroll
      for (int e = 0; e < NI; ++e) {
        double v = D00 * G[j][e];
        if (j > 0) v = fma(j * B01, G[j > 0 ? j - 1 : 0][e], v);
        if (e > 0) v = fma(e * B00, G[j][e > 0 ? e - 1 : 0], v);
        G[j + 1][e] = v;
      }
    const double cdv = hdr[3 + d], abv = hdr[d];
    const double* ex = cf + t * CFT + NR * 10;
    const double e2a = ex[0], e2b = ex[1], e2c = ex[2];
    double2* Fo = reinterpret_cast<double2*>(F + (size_t)t * St + (size_t)(job - 3 * nrw * t) * J4);
    int col = sub;  // counts down to this thread's next (c, d) column
#pragma unroll
    for (int m = 0; m < NJ - 1; ++m) {  // ket level d = m: G[c][e] = V[e][c][m]
      if (m > ld) break;
      if (m > 0) {
#pragma unroll
        for (int cc = 0; cc + m < NJ; ++cc)
#pragma unroll
          for (int e = 0; e < NI; ++e) G[cc][e] = fma(cdv, G[cc][e], G[cc + 1][e]);
      }
#pragma unroll
      for (int cc = 0; cc + m + 1 < NJ; ++cc) {
        if (cc > lc) break;
        if (col-- != 0) continue;
        col = nsub - 1;
        double u[NI], w[NI], up[NI];
#pragma unroll
        for (int e = 0; e < NI; ++e) {
          u[e] = G[cc][e];
          w[e] = e2c * G[cc + 1][e];
          if (cc > 0) w[e] = fma((double)-cc, G[cc > 0 ? cc - 1 : 0][e], w[e]);
          up[e] = 0.0;
        }
        double2* Fc = Fo + 2 * (la + 1) * (lb + 1) * (cc + (lc + 1) * m);
#pragma unroll
        for (int b = 0; b < NI - 1; ++b) {
          if (b > lb) break;
          double ud = 0.0;  // U(a-1, b)
#pragma unroll
          for (int e = 0; e + b < NI - 1; ++e) {
            const double ue = u[e], un = fma(abv, ue, u[e + 1]);  // U(a, b+1)
            if (e <= la) {
              double2 v01, v23;
              v01.x = ue;
              v01.y = e2a * u[e + 1];
              if (e > 0) v01.y = fma((double)-e, ud, v01.y);
              v23.x = e2b * un;
              if (b > 0) v23.x = fma((double)-b, up[e], v23.x);
              v23.y = w[e];
              Fc[2 * (e + (la + 1) * b)] = v01;
              Fc[2 * (e + (la + 1) * b) + 1] = v23;
            }
            w[e] = fma(abv, w[e], w[e + 1]);
            ud = ue;
            up[e] = ue;
            u[e] = un;
          }
        }
      }
    }
  }
}

// One (c, d = M) ket column of a job from its 2D table G[j][e]: the ket transfer
// in closed form, V[e][c][M] = sum_k binom(M, k) CD^(M-k) G[c+k][e], for columns
// c-1, c, c+1, then the bra transfer and the derivative factors in registers.
template <int NI, int NJ, int M>
__device__ __forceinline__ void grad_column(const double* __restrict__ G, int cc, int la, int lb, double abv,
                                            double cdv, const double* __restrict__ ex, double2* __restrict__ Fc) {
  constexpr double bin[4][4] = {{1, 0, 0, 0}, {1, 1, 0, 0}, {1, 2, 1, 0}, {1, 3, 3, 1}};
  const double e2a = ex[0], e2b = ex[1], e2c = ex[2];
  double ck[M + 1], p = 1.0;
#pragma unroll
  for (int k = M; k >= 0; --k) {
    ck[k] = bin[M][k] * p;
    p *= cdv;
  }
  const double mc = (double)-cc;
  const double* Gc = G + cc * NI;
  double u[NI], w[NI], up[NI];
#pragma unroll
  for (int e = 0; e < NI; ++e) {
    double v = 0.0, vp = 0.0, vm = 0.0;
#pragma unroll
    for (int k = 0; k <= M + 1; ++k) {  // rows c .. c + M + 1
      const double x = Gc[k * NI + e];
      if (k <= M) v = fma(ck[k <= M ? k : 0], x, v);
      if (k > 0) vp = fma(ck[k > 0 ? k - 1 : 0], x, vp);
      if (k < M) vm = fma(ck[k < M ? k + 1 : 0], x, vm);
    }
    if (cc > 0) vm = fma(ck[0], Gc[e - NI], vm);
    u[e] = v;
    w[e] = fma(mc, vm, e2c * vp);
    up[e] = 0.0;
  }
#pragma unroll
  for (int b = 0; b < NI - 1; ++b) {
    if (b > lb) break;
    double ud = 0.0;  // U(a-1, b)
#pragma unroll
    for (int e = 0; e + b < NI - 1; ++e) {
      const double ue = u[e], un = fma(abv, ue, u[e + 1]);  // U(a, b+1)
      if (e <= la) {
        double2 v01, v23;
        v01.x = ue;
        v01.y = e2a * u[e + 1];
        if (e > 0) v01.y = fma((double)-e, ud, v01.y);
        v23.x = e2b * un;
        if (b > 0) v23.x = fma((double)-b, up[e], v23.x);
        v23.y = w[e];
        Fc[2 * (e + (la + 1) * b)] = v01;
        Fc[2 * (e + (la + 1) * b) + 1] = v23;
      }
      w[e] = fma(abv, w[e], w[e + 1]);
      ud = ue;
      up[e] = ue;
      u[e] = un;
    }
  }
}

// Persistent kernel: each group of tpq threads takes work items from a
// counter until none are left.  The contracted Cartesian 2-PDM of an item
// (Gam[il][abcd]) and the stage-0 temporaries live in the group's global
// scratch slot (L2 resident); the per-tile data in shared memory.
// Per-group shared layout (doubles, every region starts on an even offset):
//   hdr[8] (AB, CD, item) | Cab | Ccd | Y | union{ reduction | tile: cf | Gp | F | S }
// F holds, per (quartet, root, direction), the 2D integral and its three
// centre derivatives interleaved: F[job * J4 + e1 * 4 + {0: I, 1: dA, 2: dB, 3: dC}],
// J4 = 4 n1d + 2: a job stride of 2 mod 4 doubles shifts each job's 16-byte
// records by an odd number of bank groups, so the jobs that a warp's lane
// segments store at once fall in different banks.
// Threads per CTA of a variant: 512 when one CTA fills the SM (128 registers
// per thread), 256 otherwise.
template <int MINB>
struct GradThreads {
  static constexpr int value = MINB == 1 ? 512 : 256;
};

template <int NAB1, int NCD1, int MINB>
__global__ void __launch_bounds__(GradThreads<MINB>::value, MINB) grad_kernel(const GradArgs a, const RysArgs ra) {
  constexpr int NR = (NAB1 + NCD1 + 1) / 2;
  constexpr int NI = NAB1 + 1, NJ = NCD1 + 1;
  extern __shared__ __align__(16) double smem_all[];
  double* tabs = smem_all;
  for (int o = threadIdx.x; o < kGTabD; o += blockDim.x) tabs[o] = a.gtab[o];
  __syncthreads();
  const int tpq = a.tpq;
  const int g = threadIdx.x / tpq;
  const int tid = threadIdx.x - g * tpq;
  double* sm = smem_all + kGTabD + (size_t)g * a.gsm;
  double* Gg = a.scratch + (size_t)(blockIdx.x * (blockDim.x / tpq) + g) * a.scr_stride;
  int* slot = reinterpret_cast<int*>(sm + 6);
  for (;;) {
  if (tid == 0) *slot = atomicAdd(a.counter, 1);
  gsync(g, tpq);
  const int item = *slot;
  if (item >= a.nitems) break;
  const int* cart = reinterpret_cast<const int*>(tabs + kGTabCart);
  const double* prim = a.prim;
  const int tot_np = a.tot_np;
  const GradItem it = a.items[item];
  const DPair& P = a.pairs[it.p];
  const DPair& Q = a.pairs[it.q];
  const int la = P.la, lb = P.lb, lc = Q.la, ld = Q.lb;
  const int nca = d_ncart(la), ncb = d_ncart(lb), ncc = d_ncart(lc), ncd = d_ncart(ld);
  const int nsa = d_ncomp(la), nsb = d_ncomp(lb), nsc = d_ncomp(lc), nsd = d_ncomp(ld);
  const int ncart4 = nca * ncb * ncc * ncd;
  const int nij = it.i1 - it.i0;   // bra contracted pairs [i0, i1)
  const int nklc = it.c1 - it.c0;  // ket contracted pairs [c0, c1)
  const int nc = nij * nklc;
  const bool multi = nc > 1;
  const int npab = P.np, npcd = Q.np;
  const int n1d = (la + 1) * (lb + 1) * (lc + 1) * (ld + 1);
  const int PAB = a.PAB, PCD = a.PCD, RW = a.RW;
  const int NT = PAB * PCD;
  const int CFT = NR * 10 + 5;  // per-quartet coefficient record (odd stride)
  double* hdr = sm;
  const int npabs = ev2(npab), npcds = ev2(npcd);     // even rows: pairs of coefficients load at once
  double* Cab = hdr + 8;                              // nij * npabs
  double* Ccd = Cab + nij * npabs;                    // nklc * npcds
  double* Y = Ccd + nklc * npcds;                     // [ij][pc][abcd] (multi only)
  int* IX = reinterpret_cast<int*>(Y + (multi ? ev2(nij * PCD * ncart4) : 0));  // [abcd] packed 2D indices
  double* U0 = reinterpret_cast<double*>(IX) + ev2((ncart4 + 1) / 2);
  // padded strides: consecutive primitive quartets fall in different bank groups
  const int Gs = ncart4 | 1;                          // Gp row (odd)
  const int J4 = 4 * n1d + 2;                          // F record of one (root, direction) job
  const int St = 3 * RW * J4 + (RW & 1 ? 0 : 2);       // F block of one quartet (= 2 mod 4)
  double* cf = U0;                                    // NT * CFT
  double* Gp = cf + ev2(NT * CFT);                    // [t][abcd] primitive 2-PDM, row stride Gs
  double* F = Gp + ev2(NT * Gs);                      // [t][rl][dir][e1][4], job stride J4, quartet stride St
  constexpr int GS = (NI * NJ) | 1;                   // 2D table of one job (odd stride), large classes only
  double* G2 = F + (size_t)NT * St;                   // [job][j][e]
  double* Gam = Gg;                                   // [il][abcd] (global scratch)
  double* Tmp = Gg + ev2(nc * ncart4);                // stage-0 temp (global scratch)
  if (tid < 3) {
    hdr[tid] = P.A[tid] - P.B[tid];
    hdr[3 + tid] = Q.A[tid] - Q.B[tid];
  }
  {
    const FDiv fab = fdiv(npab), fcd = fdiv(npcd);
    for (int o = tid; o < nij * npab; o += tpq) {
      const int ij = fq(o, fab);
      Cab[o + ij * (npabs - npab)] = a.coef[P.coef_off + (size_t)it.i0 * npab + o];
    }
    for (int o = tid; o < nklc * npcd; o += tpq) {
      const int kl = fq(o, fcd);
      Ccd[o + kl * (npcds - npcd)] = a.coef[Q.coef_off + (size_t)it.c0 * npcd + o];
    }
  }
  // ---- stage 0: contracted 2-PDM (PGet1), spherical, then -> Cartesian
  {
    const double* Dm = a.Dm;
    const size_t nbf = a.nbf;
    const int nsp4 = nsa * nsb * nsc * nsd;
    const SDiv dnc = sdiv(nc), dnsa = sdiv(nsa), dnsb = sdiv(nsb), dnsc = sdiv(nsc), dnij = sdiv(nij),
               dpi = sdiv(P.nci), dqi = sdiv(Q.nci);
    for (int o = tid; o < nc * nsp4; o += tpq) {
      int il, sa, sb, sc, ijl, ki, kk;
      const int r1 = sq(o, dnc, il), r2 = sq(r1, dnsa, sa), r3 = sq(r2, dnsb, sb), sd = sq(r3, dnsc, sc);
      const int kl = it.c0 + sq(il, dnij, ijl), ij = it.i0 + ijl;
      const int kj = sq(ij, dpi, ki), kq = sq(kl, dqi, kk);
      const int pa = P.ao_a + sa * P.nci + ki, pb = P.ao_b + sb * P.ncj + kj;
      const int pc = Q.ao_a + sc * Q.nci + kk, pd = Q.ao_b + sd * Q.ncj + kq;
      // D is symmetric: index it with the fastest-varying AO (pa, then pb) as the
      // column so that neighbouring threads read neighbouring addresses
      double x = Dm[pc * nbf + pa] * Dm[pd * nbf + pb] + Dm[pd * nbf + pa] * Dm[pc * nbf + pb];
      if (a.Ds) x += a.Ds[pc * nbf + pa] * a.Ds[pd * nbf + pb] + a.Ds[pd * nbf + pa] * a.Ds[pc * nbf + pb];
      Tmp[o] = a.cq * Dm[pb * nbf + pa] * Dm[pd * nbf + pc] - a.xq * x;
    }
    gsync(g, tpq);
    const double* Sd = tabs + kGTabSph + d_sph_off(ld);
    const double* Sc = tabs + kGTabSph + d_sph_off(lc);
    const double* Sb = tabs + kGTabSph + d_sph_off(lb);
    const double* Sa = tabs + kGTabSph + d_sph_off(la);
    // one-index transforms, ping-ponging between the two scratch buffers; s and p
    // shells are Cartesian already (identity), so their passes are skipped
    double* cur = Tmp;
    double* nxt = Gam;
    if (ld >= 2) {  // d: [il][sa][sb][sc][sd] -> [il][sa][sb][sc][cd]
      const int inner = nc * nsa * nsb * nsc;
      const SDiv din = sdiv(inner);
      for (int o = tid; o < inner * ncd; o += tpq) {
        int in;
        const int cd = sq(o, din, in);
        double s = 0;
        for (int m = 0; m < nsd; ++m) s = fma(Sd[cd + ncd * m], cur[in + inner * m], s);
        nxt[o] = s;
      }
      gsync(g, tpq);
      double* t = cur; cur = nxt; nxt = t;
    }
    if (lc >= 2) {  // c
      const int inner = nc * nsa * nsb;
      const SDiv din = sdiv(inner), dcc = sdiv(ncc);
      for (int o = tid; o < inner * ncc * ncd; o += tpq) {
        int in, cc;
        const int cd = sq(sq(o, din, in), dcc, cc);
        double s = 0;
        for (int m = 0; m < nsc; ++m) s = fma(Sc[cc + ncc * m], cur[in + inner * (m + nsc * cd)], s);
        nxt[o] = s;
      }
      gsync(g, tpq);
      double* t = cur; cur = nxt; nxt = t;
    }
    if (lb >= 2) {  // b
      const int inner = nc * nsa;
      const int outer = ncc * ncd;
      const SDiv din = sdiv(inner), dcb = sdiv(ncb);
      for (int o = tid; o < inner * ncb * outer; o += tpq) {
        int in, cb;
        const int ou = sq(sq(o, din, in), dcb, cb);
        double s = 0;
        for (int m = 0; m < nsb; ++m) s = fma(Sb[cb + ncb * m], cur[in + inner * (m + nsb * ou)], s);
        nxt[o] = s;
      }
      gsync(g, tpq);
      double* t = cur; cur = nxt; nxt = t;
    }
    if (la >= 2) {  // a
      const int outer = ncb * ncc * ncd;
      const SDiv dca = sdiv(nca);
      for (int o = tid; o < nc * nca * outer; o += tpq) {
        int il, ca;
        const int ou = sq(sq(o, dnc, il), dca, ca);
        double s = 0;
        for (int m = 0; m < nsa; ++m) s = fma(Sa[ca + nca * m], cur[il + nc * (m + nsa * ou)], s);
        nxt[o] = s;
      }
      gsync(g, tpq);
      double* t = cur; cur = nxt; nxt = t;
    }
    const SDiv dn4 = sdiv(ncart4);
    for (int o = tid; o < nc * ncart4; o += tpq) {  // transpose to [il][abcd]
      int abcd;
      const int il = sq(o, dn4, abcd);
      nxt[o] = cur[il + nc * abcd];
    }
    Gam = nxt;
    gsync(g, tpq);
  }
  double acc[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) acc[k] = 0.0;
  const int ca0 = d_ccum(la), cb0 = d_ccum(lb), cc0 = d_ccum(lc), cd0 = d_ccum(ld);
  // packed 2D-integral offsets of every Cartesian quartet: x | y << 8 | z << 16
  {
    const FDiv fca = fdiv(nca), fcb = fdiv(ncb), fcc = fdiv(ncc);
    for (int abcd = tid; abcd < ncart4; abcd += tpq) {
      const int r1 = fq(abcd, fca), ca = abcd - r1 * nca;
      const int r2 = fq(r1, fcb), cb = r1 - r2 * ncb;
      const int cd = fq(r2, fcc), cc = r2 - cd * ncc;
      const int ea = cart[ca0 + ca], eb = cart[cb0 + cb], ec = cart[cc0 + cc], ed = cart[cd0 + cd];
      int pk = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int sh = 8 * d;
        pk |= (((ea >> sh) & 255) +
               (la + 1) * (((eb >> sh) & 255) + (lb + 1) * (((ec >> sh) & 255) + (lc + 1) * ((ed >> sh) & 255))))
              << sh;
      }
      IX[abcd] = pk;
    }
  }
  for (int pcd0 = 0; pcd0 < npcd; pcd0 += PCD) {
    const int npc = min(PCD, npcd - pcd0);
    gsync(g, tpq);
    // ---- ket half-transform of the 2-PDM: Y[ij][pc][abcd] = sum_kl Ccd[kl][pc] Gam[ij,kl][abcd];
    //      a thread makes 4 consecutive pc of one (ij, abcd), each Gam load feeds 4 FMAs
    if (multi) {
      const int npc4 = (npc + 3) >> 2;
      const FDiv f4 = fdiv(ncart4), fpc = fdiv(npc4);
      for (int o = tid; o < nij * npc4 * ncart4; o += tpq) {
        const int r1 = fq(o, f4), abcd = o - r1 * ncart4, ij = fq(r1, fpc), pc0 = 4 * (r1 - ij * npc4);
        const double* gm = Gam + (size_t)ij * ncart4 + abcd;
        const double* cc = Ccd + pcd0 + pc0;
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        // (coefficients past the chunk belong to sums that are not stored)
        if (pcd0 & 1) {
          for (int klc = 0; klc < nklc; ++klc) axpy4<false>(cc + klc * npcds, gm[(size_t)nij * klc * ncart4], s);
        } else {
          for (int klc = 0; klc < nklc; ++klc) axpy4<true>(cc + klc * npcds, gm[(size_t)nij * klc * ncart4], s);
        }
        double* y = Y + abcd + ncart4 * (pc0 + PCD * ij);
        y[0] = s[0];
        if (pc0 + 1 < npc) y[ncart4] = s[1];
        if (pc0 + 2 < npc) y[2 * ncart4] = s[2];
        if (pc0 + 3 < npc) y[3 * ncart4] = s[3];
      }
    }
    for (int pab0 = 0; pab0 < npab; pab0 += PAB) {
      const int npa = min(PAB, npab - pab0);
      const int nt = npa * npc;
      const FDiv fnpa = fdiv(npa);
      gsync(g, tpq);
      // ---- (1) roots: one (primitive quartet, root) per thread
      for (int job = tid; job < nt * NR; job += tpq) {
        const int t = job / NR, r = job - t * NR;
        const int pc = fq(t, fnpa), pa = t - pc * npa;
        const int ia = P.prim_off + pab0 + pa, ic = Q.prim_off + pcd0 + pc;
        const double zeta = prim[ia], eta = prim[ic];
        const double px = prim[2 * tot_np + ia], py = prim[3 * tot_np + ia], pz = prim[4 * tot_np + ia];
        const double qx = prim[2 * tot_np + ic], qy = prim[3 * tot_np + ic], qz = prim[4 * tot_np + ic];
        double zei, rzei;  // 1 / (zeta + eta) and its root
        recip_root(zeta + eta, zei, rzei);
        const double rho = zeta * eta * zei;
        const double dx = px - qx, dy = py - qy, dz = pz - qz;
        const double T = rho * (dx * dx + dy * dy + dz * dz);
        double x, w;
        rys_one<NR>(ra, T, r, x, w);
        const double fact = prim[tot_np + ia] * prim[tot_np + ic] * rzei;
        const double U2 = x * zei;
        double* c = cf + t * CFT + r * 10;
        c[0] = 0.5 * U2;
        c[1] = 0.5 * (1.0 - U2 * eta) * prim[7 * tot_np + ia];
        c[2] = 0.5 * (1.0 - U2 * zeta) * prim[7 * tot_np + ic];
        c[3] = px - P.A[0] - eta * U2 * dx;
        c[4] = py - P.A[1] - eta * U2 * dy;
        c[5] = pz - P.A[2] - eta * U2 * dz;
        c[6] = qx - Q.A[0] + zeta * U2 * dx;
        c[7] = qy - Q.A[1] + zeta * U2 * dy;
        c[8] = qz - Q.A[2] + zeta * U2 * dz;
        c[9] = w * fact;
        if (r == 0) {
          double* e = cf + t * CFT + NR * 10;
          e[0] = 2.0 * prim[5 * tot_np + ia];         // 2 alpha
          e[1] = 2.0 * prim[6 * tot_np + ia];         // 2 beta
          e[2] = 2.0 * prim[5 * tot_np + ic];         // 2 gamma
        }
      }
      // (no barrier: the primitive 2-PDM below reads neither the roots' records nor
      // anything they overwrite, so both stages share one phase)
      // ---- (3) primitive 2-PDM (Tcrtnc): bra half-transform of Y (a thread makes 4
      //      consecutive pa of one (pc, abcd), each Y load feeds 4 FMAs), or the single
      //      contraction coefficient times the contracted 2-PDM
      {
        const int npa4 = (npa + 3) >> 2;
        const FDiv f4 = fdiv(ncart4), fpa = fdiv(npa4);
        for (int o = tid; o < npa4 * npc * ncart4; o += tpq) {
          const int r1 = fq(o, f4), abcd = o - r1 * ncart4, pc = fq(r1, fpa), pa0 = 4 * (r1 - pc * npa4);
          double s[4] = {0.0, 0.0, 0.0, 0.0};
          const double* ca = Cab + pab0 + pa0;
          if (multi) {
            const double* y = Y + abcd + ncart4 * pc;
            if (pab0 & 1) {
              for (int ij = 0; ij < nij; ++ij) axpy4<false>(ca + ij * npabs, y[ncart4 * PCD * ij], s);
            } else {
              for (int ij = 0; ij < nij; ++ij) axpy4<true>(ca + ij * npabs, y[ncart4 * PCD * ij], s);
            }
          } else {
            axpy4<false>(ca, Gam[abcd] * Ccd[pcd0 + pc], s);
          }
          double* gp = Gp + (size_t)(pa0 + npa * pc) * Gs + abcd;
          gp[0] = s[0];
          if (pa0 + 1 < npa) gp[Gs] = s[1];
          if (pa0 + 2 < npa) gp[2 * Gs] = s[2];
          if (pa0 + 3 < npa) gp[3 * Gs] = s[3];
        }
      }
      gsync(g, tpq);
      for (int r0 = 0; r0 < NR; r0 += RW) {
        const int nrw = min(RW, NR - r0);
        const FDiv fnrw = fdiv(nrw);
        // ---- (2) 2D integrals of every (quartet, root, direction) job:
        //      2D recursion  G[e][j+1] = D00 G[e][j] + j B01 G[e][j-1] + e B00 G[e-1][j];
        //      ket 2D-level HRR (HRR2Db):  V[e][c][0] = G[e][c],
        //        V[e][c][d+1] = V[e][c+1][d] + CD V[e][c][d];
        //      bra 2D-level HRR (HRR2Da):
        //        U(a,0) = V[a][c][d],  U(a,b+1) = U(a+1,b) + AB U(a,b);
        //      derivative factors (Rys2Dg): F = U, dA = 2alpha U(a+1,b) - a U(a-1,b),
        //        dB = 2beta U(a,b+1) - b U(a,b-1), dC = the same transfer of
        //        W[a] = 2gamma V[a][c+1][d] - c V[a][c-1][d]
        if constexpr (NI * NJ <= kGradJobMax) {
          grad_jobs_thread<NI, NJ, NR>(cf, CFT, hdr, F, nt, nrw, r0, la, lb, lc, ld, J4, St, fnrw, tid, tpq);
        } else {
          // the recursion by one NI-lane segment of a warp per job (32/NI jobs per warp; lane e
          // holds the row G[e][0..NJ-1] and takes G[e-1][j] from its neighbour) into the
          // job's table, then one thread per job and (c, d) column
          constexpr int JPW = 32 / NI;  // jobs per warp
          const int njobs = nt * nrw * 3;
          const int lane = tid & 31;
          const int seg = lane / NI, e = lane - seg * NI;  // seg >= JPW: spare lanes
          const int lup = (lane + 31) & 31;
          for (int jb = (tid >> 5) * JPW; jb < njobs; jb += (tpq >> 5) * JPW) {  // warp-uniform trip count
            const bool valid = seg < JPW && jb + seg < njobs;
            const int job = min(jb + seg, njobs - 1);
            const int d = job % 3, tr = job / 3, t = fq(tr, fnrw), rl = tr - t * nrw, r = r0 + rl;
            const double* c = cf + t * CFT + r * 10;
            const double B00 = c[0], B10 = c[1], B01 = c[2], C00 = c[3 + d], D00 = c[6 + d];
            // column 0 by the recursion over e: G[i+1][0] = C00 G[i][0] + i B10 G[i-1][0]
            double gm1 = 0.0, g0 = d == 2 ? c[9] : 1.0;
            for (int i = 0; i < e; ++i) {
              const double gn = fma(i * B10, gm1, C00 * g0);
              gm1 = g0;
              g0 = gn;
            }
            double* Go = G2 + (size_t)job * GS + e;
            double L = g0, Lm = 0.0;
            if (valid) Go[0] = L;
#pragma unroll
            for (int j = 0; j < NJ - 1; ++j) {
              const double up = __shfl_sync(0xffffffffu, L, lup);  // G[e-1][j]
              double v = D00 * L;
              if (j > 0) v = fma(j * B01, Lm, v);
              if (e > 0) v = fma(e * B00, up, v);
              Lm = L;
              L = v;
              if (valid) Go[(j + 1) * NI] = v;
            }
          }
          gsync(g, tpq);
          const int ncol = (lc + 1) * (ld + 1);
          const FDiv fjobs = fdiv(njobs), flc = fdiv(lc + 1);
          for (int w = tid; w < njobs * ncol; w += tpq) {
            const int col = fq(w, fjobs), job = w - col * njobs;
            const int m = fq(col, flc), cc = col - m * (lc + 1);
            const int d = job % 3, tr = job / 3, t = fq(tr, fnrw);
            const double* ex = cf + t * CFT + NR * 10;
            double2* Fc = reinterpret_cast<double2*>(F + (size_t)t * St + (size_t)(job - 3 * nrw * t) * J4) +
                          2 * (la + 1) * (lb + 1) * col;
            const double* Gj = G2 + (size_t)job * GS;
            const double abv = hdr[d], cdv = hdr[3 + d];
            switch (m) {
              case 0: grad_column<NI, NJ, 0>(Gj, cc, la, lb, abv, cdv, ex, Fc); break;
              case 1: grad_column<NI, NJ, 1>(Gj, cc, la, lb, abv, cdv, ex, Fc); break;
              case 2: grad_column<NI, NJ, 2>(Gj, cc, la, lb, abv, cdv, ex, Fc); break;
              case 3: grad_column<NI, NJ, 3>(Gj, cc, la, lb, abv, cdv, ex, Fc); break;
            }
          }
        }
        gsync(g, tpq);
        // ---- (4) Assg1: sum over Cartesian components and roots; consecutive threads
        //      take consecutive primitive quartets of one component block (the components
        //      of centre A for la = 1, 2, with those of B where possible; those of centre
        //      B when la = 0, which puts B first in the component order with unit stride)
        const int lblk = la > 0 ? la : lb;
        // both bra shells of (p p| in one block where the ket components still give every
        // thread something to do ((p d| that way: 24 instead of 12 values per direction
        // in registers, and class (4, 3) of the 460-function gradient 222 instead of
        // 180 ms)
        const int nket = ncc * ncd;
        const bool two = la == 1 && lb == 1 && nt * nket >= tpq;
        if (NAB1 == 3 && two) {
          assg1_block<1, 1>(F, Gp, IX, nt, nket, St, Gs, J4, nrw, tid, tpq, acc);
        } else if (lblk == 1) {
          assg1_block<1, 0>(F, Gp, IX, nt, ncart4 / 3, St, Gs, J4, nrw, tid, tpq, acc);
        } else if (lblk == 2) {
          assg1_block<2, 0>(F, Gp, IX, nt, ncart4 / 6, St, Gs, J4, nrw, tid, tpq, acc);
        } else {
          const FDiv fnt = fdiv(nt);
          for (int w = tid; w < nt * ncart4; w += tpq) {
            const int abcd = fq(w, fnt), t = w - abcd * nt;
            const double gm = Gp[t * Gs + abcd];
            if (gm == 0.0) continue;
            const int pk = IX[abcd];
            const int i0 = 4 * (pk & 255), i1 = J4 + 4 * ((pk >> 8) & 255), i2 = 2 * J4 + 4 * (pk >> 16);
            const double* Fb = F + (size_t)t * St;
            for (int rl = 0; rl < nrw; ++rl, Fb += 3 * J4) {
              const double2 x01 = *reinterpret_cast<const double2*>(Fb + i0);
              const double2 x23 = *reinterpret_cast<const double2*>(Fb + i0 + 2);
              const double2 y01 = *reinterpret_cast<const double2*>(Fb + i1);
              const double2 y23 = *reinterpret_cast<const double2*>(Fb + i1 + 2);
              const double2 z01 = *reinterpret_cast<const double2*>(Fb + i2);
              const double2 z23 = *reinterpret_cast<const double2*>(Fb + i2 + 2);
              const double gyz = gm * y01.x * z01.x, gxz = gm * x01.x * z01.x, gxy = gm * x01.x * y01.x;
              acc[0] = fma(gyz, x01.y, acc[0]);
              acc[1] = fma(gxz, y01.y, acc[1]);
              acc[2] = fma(gxy, z01.y, acc[2]);
              acc[3] = fma(gyz, x23.x, acc[3]);
              acc[4] = fma(gxz, y23.x, acc[4]);
              acc[5] = fma(gxy, z23.x, acc[5]);
              acc[6] = fma(gyz, x23.y, acc[6]);
              acc[7] = fma(gxz, y23.y, acc[7]);
              acc[8] = fma(gxy, z23.y, acc[8]);
            }
          }
        }
        // the next wave overwrites F; after the last wave the next tile (or chunk, or the
        // final reduction) starts with its own barrier
        if (r0 + RW < NR) gsync(g, tpq);
      }  // root waves
    }
  }
  gsync(g, tpq);
  // ---- reduce over the group, distribute to atoms (Distg1)
  double* red = U0;  // tpq/32 * 9 doubles (<= 144)
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    double v = acc[k];
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0) red[(tid >> 5) * 9 + k] = v;
  }
  gsync(g, tpq);
  if (tid < 9) {
    double v = 0.0;
    for (int w = 0; w < tpq / 32; ++w) v += red[w * 9 + tid];
    v *= it.scale;
    const int X = tid / 3, d = tid % 3;
    const int atom = X == 0 ? P.atom_a : X == 1 ? P.atom_b : Q.atom_a;
    atomicAdd(&a.grad[3 * atom + d], v);
    atomicAdd(&a.grad[3 * Q.atom_b + d], -v);  // translational invariance
  }
  gsync(g, tpq);
  }  // work items
}

template <int MINB, int A, int B>
GradFn grad_fn() {
  if (!smem_attr_once((const void*)grad_kernel<A, B, MINB>, 227 * 1024)) return nullptr;
  return grad_kernel<A, B, MINB>;
}
template <int MINB, int A>
GradFn grad_fn_b(int b) {
  switch (b) {
    case 1: return grad_fn<MINB, A, 1>();
    case 2: return grad_fn<MINB, A, 2>();
    case 3: return grad_fn<MINB, A, 3>();
    case 4: return grad_fn<MINB, A, 4>();
    case 5: return grad_fn<MINB, A, 5>();
    case 6: return grad_fn<MINB, A, 6>();
    case 7: return grad_fn<MINB, A, 7>();
  }
  return nullptr;
}
}  // namespace mg
