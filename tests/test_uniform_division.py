"""The corrected product that replaces divisions by launch constants (csrc/bk_device.cuh, div_uniform)
against the IEEE float32 quotient, restated in numpy: q = a rec, r = a - q d exactly (a float64 holds
the 48-bit product and, by cancellation, the difference), q + r rec rounded once."""
import numpy as np
import pytest

from baking_b200.config import DingConfig, MaterialConfig

f32 = np.float32


def div_uniform(a, d):
    rec = f32(1.0) / f32(d)
    q = (a * rec).astype(f32)
    r = (a.astype(np.float64) - q.astype(np.float64) * np.float64(d)).astype(f32)
    out = (q.astype(np.float64) + r.astype(np.float64) * np.float64(rec)).astype(f32)
    return np.where(np.abs(q) <= f32(3.4028235e38), out, q)


def divisors():
    m, k = MaterialConfig(), DingConfig().temperature_knots_k
    mu, lam = f32(m.shear_modulus), f32(m.lame_lambda)
    out = [f32(3.0), f32(2.0) * mu, f32(2.0) * mu + f32(3.0) * lam] + [f32(b) - f32(a) for a, b in zip(k, k[1:])]
    return out + [f32(1.0 / r) for r in (24, 32, 40, 48, 64, 96, 100, 128, 192, 256)] + [f32(0.025)]


@pytest.mark.parametrize("d", divisors(), ids=lambda d: repr(float(d)))
def test_corrected_product_is_the_quotient(d):
    rng = np.random.default_rng(0)
    mantissas = np.arange(2 ** 23, 2 ** 24, 3, dtype=np.int64).astype(f32) * f32(2.0 ** -23)  # a third of a binade
    spread = (rng.standard_normal(400_000) * 10.0 ** rng.uniform(-12, 8, 400_000)).astype(f32)
    for a in (mantissas, -spread, np.array([0.0, -0.0, np.inf, -np.inf, np.nan], f32)):
        with np.errstate(invalid="ignore", over="ignore"):
            np.testing.assert_array_equal(div_uniform(a, d), a / f32(d))
