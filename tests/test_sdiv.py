"""The kernels' corrected run-time division (SDiv in
openmolcas_b200/csrc/kern_common.cuh): m = floor(2^32 / n) (2^32 - 1 for n = 1),
q = umulhi(o, m), one step up when o - q n >= n.  Exact for every o < 2^32."""
import numpy as np

MASK = (1 << 32) - 1


def sq(o, n):
    m = MASK if n == 1 else MASK // n + (MASK % n == n - 1)
    q = (o * m) >> 32
    r = o - q * n
    assert 0 <= r < 2 * n
    return (q + 1, r - n) if r >= n else (q, r)


def test_exact_over_the_whole_range():
    rng = np.random.default_rng(5)
    ns = list(range(1, 300)) + [1 << k for k in range(32)] + rng.integers(1, MASK, 500).tolist()
    for n in ns:
        os_ = [0, 1, n - 1, n, n + 1, 2 * n - 1, MASK, MASK - 1, MASK // n * n, MASK // n * n - 1]
        for o in os_ + rng.integers(0, MASK, 20).tolist():
            if 0 <= o <= MASK:
                assert sq(o, n) == divmod(o, n), (o, n)
