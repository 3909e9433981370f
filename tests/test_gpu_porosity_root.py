"""The coupled end-state porosity solve against roots and predictions in 80-bit arithmetic, over plastic
states with porosities of 0.001 to 0.9: the returned float32 porosity is the rounded root (half a unit in
the last place and the solve's 1e-12), and the prediction evaluated at it, of which the reported
consistency is made, is exact to the overstress root's 1e-12 test."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
L = np.longdouble


def prediction(n, q, p, d, h, e, Vp, n0):
    a = L(2.25) / (np.log(n) ** 2 * (L(3.5) * n + 1))
    r = np.zeros_like(n)
    over = q + a * p > 1
    for _ in range(80):
        u, v = 1 + d * r, 1 + h * a * r
        step = (r + 1 - q / u ** 2 - a * p / v ** 2) / (1 + 2 * d * q / u ** 3 + 2 * h * a * a * p / v ** 3)
        r = np.where(over, r - step, 0)
    return Vp * np.exp(e * (1 - 1 / (1 + h * a * r))) - 1 + n0


@pytest.mark.parametrize("low,high", [(0.001, 0.05), (0.05, 0.5), (0.5, 0.9)])
def test_root_and_prediction(low, high):
    from baking_b200.physics.materials.porous_return import SolvePorosity
    rng = np.random.default_rng(3)
    count, n0 = 4000, np.float32(0.2)
    porosity = np.exp(rng.uniform(np.log(low), np.log(high), count)).astype(np.float32)
    a = 2.25 / (np.log(porosity.astype(np.float64)) ** 2 * (3.5 * porosity + 1))
    q = rng.uniform(0, 3, count).astype(np.float32)
    p = (10 ** rng.uniform(-2, 1.5, count) / a).astype(np.float32)
    q = np.where(q + a * p > 1.001, q, q + 1.1).astype(np.float32)  # past the yield surface
    d = (10 ** rng.uniform(-6, 0, count)).astype(np.float32)
    h = (d * rng.uniform(0.3, 3, count)).astype(np.float32)
    e = (rng.uniform(-0.3, 0.3, count) * porosity).astype(np.float32)
    Vp = 1.0 - float(n0) + porosity.astype(np.float64)
    got, predicted = SolvePorosity(q, p, d, h, e, Vp, float(n0))
    got, predicted = got.cpu().numpy(), predicted.cpu().numpy()
    args = [x.astype(L) for x in (q, p, d, h, e, Vp)] + [L(n0)]
    # a state whose prediction stays above 1 has no porosity
    some = Vp * np.exp(e.astype(np.float64)) - 1.0 + float(n0) < 1.0 - 1e-9
    assert some.mean() > 0.5
    delta = np.spacing(got).astype(L) / 2 + L(1e-12)
    with np.errstate(divide="ignore", invalid="ignore"):  # states without a porosity end at 1
        below, above = (got + side * delta - prediction(got + side * delta, *args) for side in (-1, 1))
        at = prediction(got.astype(L), *args)
    assert (below * above <= 0)[some].all()
    assert (np.abs(predicted - at) <= 1e-12)[some].all()
