"""Pieces of the Rys kernels' arithmetic, compiled from their headers and run on
the device: the divisions, the reciprocal and reciprocal root of the primitive
quartets, and one ket column of the gradient's 2D integrals (transfer in closed
form) against the recurrences it stands for."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.test_sdiv import MASK, compile_header, edge_pairs

pytestmark = pytest.mark.gpu

DRIVER = r"""
#include "grad_kernel.cuh"
__global__ void k_div(int k, const unsigned* o, const unsigned* n, unsigned* q, unsigned* r, unsigned* f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  int rem;
  q[i] = (unsigned)mg::sq((int)o[i], mg::sdiv(n[i]), rem);
  r[i] = (unsigned)rem;
  f[i] = mg::fq(o[i], mg::fdiv(n[i]));
}
__global__ void k_recip(int k, const double* x, double* xi, double* rxi) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < k) mg::recip_root(x[i], xi[i], rxi[i]);
}
// all (c, d) columns of one job: F[(a + (la+1)(b + (lb+1)(c + (lc+1) d))) 4 + {I, dA, dB, dC}]
template <int NI, int NJ>
__global__ void k_columns(const double* G, int la, int lb, int lc, int ld, double ab, double cd, const double* ex,
                          double* F) {
  for (int d = 0; d <= ld; ++d)
    for (int c = 0; c <= lc; ++c) {
      double2* f = reinterpret_cast<double2*>(F) + 2 * (la + 1) * (lb + 1) * (c + (lc + 1) * d);
      if (d == 0) mg::grad_column<NI, NJ, 0>(G, c, la, lb, ab, cd, ex, f);
      if (d == 1) mg::grad_column<NI, NJ, 1>(G, c, la, lb, ab, cd, ex, f);
      if (d == 2) mg::grad_column<NI, NJ, 2>(G, c, la, lb, ab, cd, ex, f);
      if (d == 3) mg::grad_column<NI, NJ, 3>(G, c, la, lb, ab, cd, ex, f);
    }
}
extern "C" int run_div(int k, const unsigned* o, const unsigned* n, unsigned* q, unsigned* r, unsigned* f) {
  k_div<<<(k + 255) / 256, 256>>>(k, o, n, q, r, f);
  return cudaDeviceSynchronize();
}
extern "C" int run_recip(int k, const double* x, double* xi, double* rxi) {
  k_recip<<<(k + 255) / 256, 256>>>(k, x, xi, rxi);
  return cudaDeviceSynchronize();
}
extern "C" int run_columns(int ni, int nj, const double* G, int la, int lb, int lc, int ld, double ab, double cd,
                           const double* ex, double* F) {
  if (ni == 5 && nj == 5) k_columns<5, 5><<<1, 1>>>(G, la, lb, lc, ld, ab, cd, ex, F);
  else if (ni == 6 && nj == 4) k_columns<6, 4><<<1, 1>>>(G, la, lb, lc, ld, ab, cd, ex, F);
  else if (ni == 4 && nj == 8) k_columns<4, 8><<<1, 1>>>(G, la, lb, lc, ld, ab, cd, ex, F);
  else return -1;
  return cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return compile_header(tmp_path_factory.mktemp("kern"), DRIVER)


def ptr(t):
    return C.c_void_p(t.data_ptr())


def test_divisions_on_the_device(lib):
    for limit in (lambda n: MASK, lambda n: MASK // n):
        o, n = edge_pairs(limit)
        dev = [torch.from_numpy(x.astype(np.uint32).view(np.int32)).cuda() for x in (o, n)]
        q, r, f = (torch.zeros_like(dev[0]) for _ in range(3))
        assert lib.run_div(C.c_int(o.size), *[ptr(t) for t in dev + [q, r, f]]) == 0
        q, r, f = (t.cpu().numpy().view(np.uint32) for t in (q, r, f))
        assert np.array_equal(q, o // n) and np.array_equal(r, o % n)
        ok = o * n <= MASK
        assert ok.any() and np.array_equal(f[ok], (o // n)[ok])


def test_reciprocal_and_root(lib):
    """Sums of two exponents over eleven decades and around powers of two, against
    80-bit values.  rsqrt is within one unit in the last place; its square, within
    2^-50.6, leaves the Newton step's final rounding as the only error of the
    reciprocal: half a unit.  (1e-3: the reference's own resolution.)"""
    assert np.finfo(np.longdouble).nmant >= 63
    rng = np.random.default_rng(7)
    near = np.outer(1.0 + np.arange(-8, 9) * 2.0 ** -52, np.ldexp(1.0, np.arange(-10, 27))).ravel()
    x = np.concatenate([10.0 ** rng.uniform(-3, 8, 1_000_000), near])
    d = torch.from_numpy(x).cuda()
    xi, rxi = torch.zeros_like(d), torch.zeros_like(d)
    assert lib.run_recip(C.c_int(x.size), ptr(d), ptr(xi), ptr(rxi)) == 0
    xl = x.astype(np.longdouble)
    for got, exact, bound in ((xi, 1 / xl, 0.5), (rxi, 1 / np.sqrt(xl), 1.0)):
        got = got.cpu().numpy()
        err = np.abs((got.astype(np.longdouble) - exact) / np.spacing(got))
        print(f"largest error {float(err.max()):.4f} units in the last place")
        assert err.max() <= bound + 1e-3


@pytest.mark.parametrize("ni,nj,la,lb,lc,ld", [(5, 5, 2, 1, 2, 1), (5, 5, 1, 2, 1, 2), (5, 5, 3, 0, 0, 3),
                                               (6, 4, 2, 2, 2, 0), (4, 8, 1, 1, 3, 3)])
def test_ket_columns_against_the_recurrences(lib, ni, nj, la, lb, lc, ld):
    """V(c, d+1) = V(c+1, d) + CD V(c, d) and U(a, b+1) = U(a+1, b) + AB U(a, b), the
    derivative factors 2x I(l+1) - l I(l-1).  The same recurrences over absolute
    values bound the sums; every value is within 32 operations of its inputs."""
    rng = np.random.default_rng(ni * 100 + nj * 10 + ld)
    G = rng.standard_normal((nj, ni))
    ab, cd = 1.3, -0.7
    ex = np.array([0.9, 2.1, 0.4])

    def columns(G, ab, cd, s):
        V = {(c, 0): G[c] for c in range(nj)}
        for d in range(ld):
            for c in range(nj - d - 1):
                V[c, d + 1] = V[c + 1, d] + cd * V[c, d]

        def bra(v):
            U = {(a, 0): v[a] for a in range(ni)}
            for b in range(lb + 1):
                for a in range(ni - b - 1):
                    U[a, b + 1] = U[a + 1, b] + ab * U[a, b]
            return U
        F = np.zeros((ld + 1, lc + 1, lb + 1, la + 1, 4))
        for d in range(ld + 1):
            for c in range(lc + 1):
                U = bra(V[c, d])
                W = bra(ex[2] * V[c + 1, d] + s * c * (V[c - 1, d] if c else 0.0 * V[c, d]))
                for b in range(lb + 1):
                    for a in range(la + 1):
                        F[d, c, b, a] = (U[a, b], ex[0] * U[a + 1, b] + s * a * U.get((a - 1, b), 0.0),
                                         ex[1] * U[a, b + 1] + s * b * U.get((a, b - 1), 0.0), W[a, b])
        return F
    want = columns(G, ab, cd, -1.0)
    scale = columns(np.abs(G), abs(ab), abs(cd), 1.0)
    dG, dex = torch.from_numpy(G).cuda(), torch.from_numpy(ex).cuda()
    F = torch.full(want.shape, float("nan"), dtype=torch.float64, device="cuda")
    assert lib.run_columns(ni, nj, ptr(dG), la, lb, lc, ld, C.c_double(ab), C.c_double(cd), ptr(dex), ptr(F)) == 0
    assert (np.abs(F.cpu().numpy() - want) <= 32 * 2.0 ** -53 * scale).all()
