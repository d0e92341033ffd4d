"""The Boys functions of every order as the class kernels evaluate them, FP64
and FP32, and their reciprocal square root, against extended precision."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(m, t):
    """F_0 .. F_m: the convergent series, and beyond 60 the upward recursion
    from sqrt(pi / T) / 2 (erfc(sqrt(60)) is 6e-28)."""
    t = t.astype(np.longdouble)
    far = t > 60
    out = np.empty((len(t), m + 1), dtype=np.longdouble)
    near, x = t[~far], t[far]
    for k in range(m + 1):
        term = np.full_like(near, 1) / (2 * k + 1)
        total = term.copy()
        for j in range(1, 400):
            term = term * 2 * near / (2 * k + 2 * j + 1)
            total += term
        out[~far, k] = np.exp(-near) * total
    f = np.sqrt(np.longdouble('3.14159265358979323846264338327950288') / x) / 2
    for k in range(m + 1):
        out[far, k] = f
        f = ((2 * k + 1) * f - np.exp(-x)) / (2 * x)
    return out


@pytest.mark.parametrize('fp32', [0, 1])
@pytest.mark.parametrize('m', range(13))
def test_every_order_to_its_rounding(m, fp32):
    """On both sides of the table's end (T = 40), on its interval borders and far
    out.  In units of the rounding error u: at most 4 from the root (2 ulp of
    rsqrtf, 3e-16 of the FP64 step) or the polynomial and 3 from the scaling, then
    3 for each order of the recursion (product and sum, factor, product)."""
    from veloxchem_b200 import _native as nat
    rng = np.random.default_rng(m)
    t = np.concatenate([[0.0, 1e-12, 0.25, 0.75, 39.75, 39.99, 40.0, 40.01], np.arange(0, 40, 0.25),
                        rng.uniform(0, 40, 4000), 10**rng.uniform(-6, 1.6, 1000), rng.uniform(40, 60, 2000),
                        rng.uniform(60, 500, 2000), 10**rng.uniform(2, 5, 500)])
    if fp32:
        t = t.astype(np.float32).astype(np.float64)
    got = np.empty((len(t), m + 1))
    nat.check(nat.lib().vlx_b200_boys_orders_device(0, m, fp32, len(t), nat.dptr(t), nat.dptr(got)), 'boys_orders')
    want = _exact(m, t)
    u = 2.0**-24 if fp32 else 2.0**-53
    # beyond the smallest normal float the FP32 values are subnormal or zero
    normal = want > 1e-37 if fp32 else np.ones_like(want, dtype=bool)
    err = np.where(normal, np.abs((got - want) / want), 0).astype(np.float64)
    assert np.max(err) < (7 + 3 * m) * u, (np.max(err) / u, t[np.argmax(np.max(err, axis=1))])


def test_reciprocal_root_to_its_bound():
    """Over the exponent sums and Boys arguments that occur, and far beyond."""
    from veloxchem_b200 import _native as nat
    rng = np.random.default_rng(1)
    x = np.concatenate([10**rng.uniform(-3, 8, 20000), 10**rng.uniform(-30, 30, 5000), rng.uniform(1, 4, 20000),
                        2.0**np.arange(-40, 40), np.nextafter(4.0**np.arange(-20, 20), np.inf)])
    got = np.empty_like(x)
    nat.check(nat.lib().vlx_b200_rsqrt_device(0, len(x), nat.dptr(x), nat.dptr(got)), 'rsqrt')
    want = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.max(np.abs((got - want) / want)) < 3e-16
