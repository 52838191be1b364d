"""The packed Fourier projection's |F| and A / |F| (project() in
csrc/ptycho_wave.cuh), restated in NumPy: one reciprocal square root of bounded
error, Newton steps whose residuals are single fused multiply-adds. Whatever the
reciprocal square root returns within its documented error (2^-22.9), the root is
at most one ulp from the correctly rounded one, and equal to it but for values next
to a tie; so is the quotient."""

import numpy as np
import pytest

f32 = np.float32


def fma(a, b, c):
    """a b + c in float32 with one rounding: the product is exact in float64, the sum
    is rounded to odd there and then to float32."""
    p, c = a.astype(np.float64) * b.astype(np.float64), c.astype(np.float64)
    s = p + c
    t = s - p
    e = (p - (s - t)) + (c - t)
    odd = s.view(np.int64) & 1
    step = np.nextafter(s, np.where(e > 0, np.inf, -np.inf))
    return np.where((e != 0) & (odd == 0), step, s).astype(f32)


def project(s, amp, rel):
    """(|F|, A / |F|) from s = |F|^2 with a reciprocal root off by the factor 1 + rel."""
    half = np.full_like(s, 0.5)
    y = (1.0 / np.sqrt(s.astype(np.float64)) * (1.0 + rel)).astype(f32)
    a0 = s * y
    e = fma(-a0, a0, s)
    a = fma(half * y, e, a0)
    y1 = fma(y, fma(-a, y, np.ones_like(s)), y)
    q0 = amp * y1
    return a, fma(fma(-q0, a, amp), y1, q0)


@pytest.mark.parametrize("rel", [-(2.0 ** -22.9), 0.0, 2.0 ** -22.9, None])
def test_root_and_quotient(rel):
    rng = np.random.default_rng(3)
    n = 400_000
    s = (rng.uniform(1.0, 4.0, n) * 2.0 ** rng.integers(-90, 90, n)).astype(f32)
    amp = (rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-20, 20, n)).astype(f32)
    if rel is None:
        rel = rng.uniform(-1.0, 1.0, n) * 2.0 ** -22.9
    a, q = project(s, amp, rel)
    root = np.sqrt(s)  # correctly rounded
    quotient = amp / root
    for got, want in ((a, root), (q, quotient)):
        ulps = np.abs(got.view(np.int32).astype(np.int64) - want.view(np.int32))
        assert ulps.max() <= 1
        assert np.count_nonzero(ulps) <= 1e-4 * n
