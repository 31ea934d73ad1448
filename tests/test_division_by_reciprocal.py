"""div_by of dev_common.cuh (a / s from the correctly rounded 1/s and one
residual correction, Markstein 1990) against IEEE f32 division, the operations
restated on the CPU: f32 products are exact in f64, and the fused additions
are taken in extended precision before the one rounding to f32.  The kernels
divide the components of a vector by its length, so |a| <= s; lengths cover
the range normalize() corrects in, and components down to 2^-60 of it."""
import numpy as np
import pytest

f32, f64, wide = np.float32, np.float64, np.longdouble


def div_by(a, s, r):
    q = (a * r).astype(f32)
    residual = (wide(a) - wide(f64(q) * f64(s))).astype(f32)  # exact: a - q s needs at most 24 bits
    return (wide(q) + wide(f64(residual) * f64(r))).astype(f32)


@pytest.mark.parametrize("seed", range(4))
def test_quotients_equal_ieee_division(seed):
    rng = np.random.default_rng(seed)
    n = 1 << 20
    s = np.ldexp(rng.uniform(1, 2, n), rng.integers(-49, 50, n)).astype(f32)
    a = (s * np.ldexp(rng.uniform(-1, 1, n), -rng.integers(0, 60, n))).astype(f32)
    a[: n // 4] = (s * rng.uniform(-1, 1, n))[: n // 4].astype(f32)
    a[: 64], s[: 64] = s[: 64], s[: 64]                                  # a / a
    s[64:128] = np.nextafter(f32(2), f32(0))                             # mantissa of all ones
    r = (f32(1) / s).astype(f32)
    want = (a / s).astype(f32)
    got = div_by(a, s, r)
    assert np.array_equal(got, want)
