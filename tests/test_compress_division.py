"""The division of the cache write: q0 = RN(x r), rem = RN(x - q0 d), q = RN(q0 + rem r) with r = RN(1 / d)
equals the IEEE quotient x / d for every pair of 24-bit significands.

Scaled to x, d in [1, 2), the value before the last rounding is v = x/d + (q0 - x/d)(1 - d r) + (error of rem) r with
|1 - d r| <= d 2^-25.  It can round another way than x/d only if a midpoint of two neighbouring floats lies
as near to x/d as v does:

  x <  d: the floats are 2^-24 apart and |q0 - x/d| <= (x + 1) 2^-25.  rem is a multiple of 2^-47, exact below 2^-23
          and else off by 2^-47.  A midpoint M 2^-25 is |j| 2^-48 / d away, where X 2^25 - M D = j for the integer
          significands X, D; so only |j| <= (x + 1) d^2 / 4, plus 2 where rem may reach 2^-23, can matter: |j| <= 5.
  x >= d: the floats are 2^-23 apart, |q0 - x/d| <= (x/2 + 1) 2^-24 and rem is exact.  A midpoint M 2^-24 is
          |j| 2^-47 / d away, X 2^24 - M D = j: only |j| <= (x/2 + 1) d^2 / 4 can matter: |j| <= 2.

For given D and j the equation has few solutions, found with the inverse of D's odd part modulo a power of two: all of
them are tried here, which covers all 2^46 pairs."""

import numpy as np
import pytest

from oracle.rq_exact import fma32


def _inverse(odd: np.ndarray, bits: int) -> np.ndarray:
    x = odd.copy()                                   # correct to 3 bits; each step doubles them
    for _ in range(4):
        x = x * (2 - odd * x)                        # modulo 2^64
    return x & np.uint64((1 << bits) - 1)


def _near_midpoints(s: int, lo: int, hi: int, below: bool):
    """The pairs (X, D) with D = 2^s * odd in [lo, hi) whose quotient is near a midpoint."""
    shift = 25 if below else 24
    d = np.arange((lo >> s) | 1, hi >> s, 2, dtype=np.uint64)
    inv = _inverse(d, shift - s)
    mod = 1 << (shift - s)
    for j in [j for j in range(-5, 6) if j % (1 << s) == 0 and (j >> s) % 2]:
        m = ((np.uint64((-(j >> s)) % mod)) * inv) & np.uint64(mod - 1)
        for first in range(1 << 24, 1 << 25, mod) if mod <= 1 << 24 else [0]:
            mm = (m + np.uint64(first)).astype(np.int64)
            dd = (d << np.uint64(s)).astype(np.int64)
            x = (mm * dd + j) >> shift
            fx, fd = x * 2.0 ** -23, dd * 2.0 ** -23
            if below:
                near = abs(j) <= (fx + 1) * fd * fd / 4 + 2 * ((fx + 1) * fd >= 4) + 1e-3
                keep = (mm > 1 << 24) & (x >= 1 << 23) & (x < dd) & near
            else:
                keep = (x >= dd) & (x < 1 << 24) & (abs(j) <= (fx / 2 + 1) * fd * fd / 4 + 1e-3)
            yield x[keep], dd[keep], mm[keep], j


def _fast(x, d):
    r = np.float32(1.0) / d
    q0 = x * r
    return fma32(fma32(-d, q0, x), r, q0)


@pytest.mark.parametrize("below", [True, False], ids=["x<d", "x>=d"])
@pytest.mark.parametrize("s", [0, 1, 2])
def test_every_quotient_near_a_midpoint(s, below):
    tried = 0
    for lo in range(1 << 23, 1 << 24, 1 << 21):
        for x, d, m, j in _near_midpoints(s, lo, lo + (1 << 21), below):
            assert bool(((x << (25 if below else 24)) - m * d == j).all())
            fx, fd = (v.astype(np.float32) * np.float32(2.0 ** -23) for v in (x, d))
            assert np.array_equal(_fast(fx, fd), fx / fd)
            tried += x.size
    assert tried > 0 or (s == 2 and not below)       # x >= d: |j| <= 2


def test_random_pairs_and_extreme_significands():
    gen = np.random.default_rng(1)
    ends = np.concatenate([np.arange(64), (1 << 23) - 1 - np.arange(64)]) + (1 << 23)
    x = np.concatenate([gen.integers(1 << 23, 1 << 24, 1 << 20), np.repeat(ends, ends.size)])
    d = np.concatenate([gen.integers(1 << 23, 1 << 24, 1 << 20), np.tile(ends, ends.size)])
    fx, fd = (v.astype(np.float32) * np.float32(2.0 ** -23) for v in (x, d))
    assert np.array_equal(_fast(fx, fd), fx / fd)
