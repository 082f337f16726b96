"""The kernels' run-time divisions as openmolcas_b200/csrc/kern_common.cuh has
them, compiled from the header and run on the host: SDiv (a multiply-high and one
correction step) exact for every o < 2^32, FDiv (no correction) for o n < 2^32,
the bound that the planners keep."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MASK = (1 << 32) - 1

DRIVER = r"""
#include "kern_common.cuh"
extern "C" void sdiv_host(int k, const unsigned* o, const unsigned* n, unsigned* q, unsigned* r) {
  for (int i = 0; i < k; ++i) {
    int rem;
    q[i] = (unsigned)mg::sq((int)o[i], mg::sdiv(n[i]), rem);
    r[i] = (unsigned)rem;
  }
}
extern "C" void fdiv_host(int k, const unsigned* o, const unsigned* n, unsigned* q) {
  for (int i = 0; i < k; ++i) q[i] = mg::fq(o[i], mg::fdiv(n[i]));
}
"""


def compile_header(tmp, source):
    """A shared library of `source`, which may include the kernels' headers."""
    src, lib = tmp / "drv.cu", tmp / "libdrv.so"
    src.write_text(source)
    r = subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                        "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(ROOT, "openmolcas_b200", "csrc"), str(src),
                        "-o", str(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return C.CDLL(str(lib))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return compile_header(tmp_path_factory.mktemp("sdiv"), DRIVER)


def divide(f, o, n, remainder):
    o, n = (np.ascontiguousarray(x, dtype=np.uint32) for x in (o, n))
    out = [np.zeros(o.size, np.uint32) for _ in range(2 if remainder else 1)]
    ptr = lambda a: a.ctypes.data_as(C.c_void_p)
    f(C.c_int(o.size), ptr(o), ptr(n), *[ptr(x) for x in out])
    return out


def edge_pairs(limit):
    """(o, n) at the edges of the quotient and at random, o <= limit(n)."""
    rng = np.random.default_rng(5)
    ns = list(range(1, 300)) + [1 << k for k in range(32)] + rng.integers(1, MASK, 500).tolist()
    o, d = [], []
    for n in ns:
        top = limit(n)
        os_ = [0, 1, n - 1, n, n + 1, 2 * n - 1, top, top - 1, top // n * n, top // n * n - 1]
        for x in os_ + rng.integers(0, top + 1, 20).tolist():
            if 0 <= x <= top:
                o.append(x)
                d.append(n)
    return np.array(o, dtype=np.uint64), np.array(d, dtype=np.uint64)


def test_exact_over_the_whole_range(lib):
    o, n = edge_pairs(lambda n: MASK)
    q, r = divide(lib.sdiv_host, o, n, True)
    assert np.array_equal(q, o // n) and np.array_equal(r, o % n)


def test_uncorrected_form_exact_below_its_bound(lib):
    o, n = edge_pairs(lambda n: MASK // n)
    (q,) = divide(lib.fdiv_host, o, n, False)
    assert np.array_equal(q, o // n)
