"""The kernels' arithmetic helpers (csrc/bk_device.cuh) on the device against numpy.

Bounds, in units of the last place of the exact value. Newton's second step leaves a residual of 2^-88,
so 1 / x is off by its last rounding: 0.51. 1 / sqrt(x) also carries the
rounding of h y, at most 2^-54 of the result: 1.5. exp's ten terms end with a rounding and 1/16 of the one
before: 0.6. Beyond the float32 range the helpers take the library's functions: 1 / x 0.51, 1 / sqrt(x) 1.0
(its documented error), exp 1.0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = np.longdouble
DIV_UNIFORM, RECIPROCAL, RSQRT, EXP_SMALL = range(4)


def device(op, a, b=None):
    import torch
    from baking_b200 import _lib
    a = torch.as_tensor(np.ascontiguousarray(a, np.float64), device="cuda")
    b = torch.ones_like(a) if b is None else torch.as_tensor(np.ascontiguousarray(b, np.float64), device="cuda")
    out = torch.empty_like(a)
    _lib.call("bk_arithmetic", op, a.numel(), a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.stream_handle())
    return out.cpu().numpy()


def ulps(got, exact):
    return np.abs(got.astype(L) - exact) / np.spacing(np.abs(exact).astype(np.float64)).astype(L)


def values(low, high, count=400_000):
    rng = np.random.default_rng(0)
    return 10.0 ** rng.uniform(low, high, count) * rng.uniform(1, 2, count)


@pytest.mark.parametrize("low,high", [(-2, 2), (-35, 35), (-300, -40), (40, 300)])
def test_reciprocal(low, high):
    x = values(low, high)
    x[::2] *= -1
    assert ulps(device(RECIPROCAL, x), 1 / x.astype(L)).max() <= 0.51


@pytest.mark.parametrize("low,high,bound", [(-2, 2, 1.5), (-35, 35, 1.5), (-300, -40, 1.0), (40, 300, 1.0)])
def test_reciprocal_root(low, high, bound):
    x = values(low, high)
    assert ulps(device(RSQRT, x), 1 / np.sqrt(x.astype(L))).max() <= bound


def test_exponential():
    x = np.random.default_rng(2).uniform(-1 / 32, 1 / 32, 400_000)
    x[:40_000] *= 1e-6
    assert ulps(device(EXP_SMALL, x), np.exp(x.astype(L))).max() <= 0.6
    x = np.random.default_rng(2).uniform(-20, 20, 400_000)
    assert ulps(device(EXP_SMALL, x), np.exp(x.astype(L))).max() <= 1.0


def test_special_values():
    x = np.array([0.0, np.inf, np.nan, 5e-324, 1e-310, -np.inf])
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(device(RECIPROCAL, x), 1.0 / x)
        np.testing.assert_array_equal(device(EXP_SMALL, np.array([0.0, -np.inf, np.inf, np.nan])),
                                      np.array([1.0, 0.0, np.inf, np.nan]))


def divisors():
    from pathlib import Path
    import baking_b200
    from tests.test_uniform_division import divisors as launch_constants
    rng = np.random.default_rng(5)
    net = np.load(Path(baking_b200.__file__).parent / "data" / "return_surrogate_box_loaf.npz")
    scales = [np.float32(v) for k in net.files if "scale" in k for v in np.ravel(net[k]) if v != 0]
    return launch_constants() + scales + [np.float32(v) for v in 10.0 ** rng.uniform(-6, 6, 24)]


def test_division_by_a_shared_divisor():
    mantissas = np.arange(2 ** 23, 2 ** 24, 5, dtype=np.int64).astype(np.float32) * np.float32(2.0 ** -23)
    rng = np.random.default_rng(0)
    spread = (rng.standard_normal(400_000) * 10.0 ** rng.uniform(-12, 8, 400_000)).astype(np.float32)
    a = np.concatenate([mantissas, -spread, np.array([0.0, np.inf, -np.inf, np.nan], np.float32)])
    tested = divisors()
    assert len(tested) > 40
    for d in tested:
        got = device(DIV_UNIFORM, a, np.full(a.shape, d))
        with np.errstate(invalid="ignore"):
            np.testing.assert_array_equal(got, (a / d).astype(np.float64), err_msg=repr(float(d)))


def test_a_divisor_of_all_ones():
    """The one kind of divisor for which the corrected product is not always the quotient: at most a unit
    in the last place off, in a handful of quotients of a binade."""
    d = np.float32(np.nextafter(np.float32(1), np.float32(0)))
    a = np.arange(2 ** 23, 2 ** 24, dtype=np.int64).astype(np.float32) * np.float32(2.0 ** -23)
    got, exact = device(DIV_UNIFORM, a, np.full(a.shape, d)), (a / d).astype(np.float64)
    assert (np.abs(got - exact) <= np.spacing(exact.astype(np.float32))).all()
    assert np.count_nonzero(got != exact) <= 16
