"""The segment weights of the piecewise-linear Laplace transform from small to very large |z h|, against the
same sums in extended precision."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _weights(x):
    """(phi1, phi2) in extended precision."""
    small = np.abs(x) < 0.5
    xs, xl = np.where(small, x, 0), np.where(small, 1, x)
    p2, f = np.zeros_like(x), np.clongdouble(1)
    c = [np.longdouble(1) / 2]
    for k in range(1, 30):
        c.append(c[-1] / (k + 2))
    for k in range(29, -1, -1):
        p2 = p2 * xs + c[k]
    ex = np.exp(xl)
    p2 = np.where(small, p2, (ex - 1 - xl) / (xl * xl))
    return np.where(small, 1 + xs * p2, (ex - 1) / xl), p2


@pytest.mark.parametrize("size", [2.0**-4, 2.0**-2, 1.0, 2.0**3, 2.0**7, 2.0**12, 2.0**17])
def test_weights(cuda, size):
    from cmpy_gb300 import engine as E

    # times and frequencies whose products are exact: what is left are the weights' own roundings
    r = np.random.default_rng(int(16 * size))
    t = np.cumsum(r.integers(1, 5, 40)) / 16.0
    g = r.standard_normal(40) + 1j * r.standard_normal(40)
    z = size * (np.arange(-12, 13) / 4.0 + 4.0) + 1j * np.where(np.arange(25) % 2, 0.0, 2.0**-6)
    got = E.laplace_t2z(t, g, z).cpu().numpy()
    zl, tl, gl = z.astype(np.clongdouble), t.astype(np.longdouble), g.astype(np.clongdouble)
    u, h = 1j * zl[:, None], np.diff(tl)[None, :]
    p1, p2 = _weights(u * h)
    ph = h * np.exp(u * tl[None, :-1])
    ref = np.sum(ph * (gl[:-1] * p2 + gl[1:] * (p1 - p2)), axis=1)
    # an exponential (2), the weights (5 each, of their own size; below |x| = 1 the closed form loses up to
    # 4 / |x|^2 of a rounding, at most 64, to the cancellation), three complex products (3 each), and the sum
    w = np.abs(ph) * (np.abs(gl[:-1]) * np.abs(p2) + np.abs(gl[1:]) * (np.abs(p1) + np.abs(p2)))
    x = np.abs(u * h)
    lost = np.where((x >= 0.25) & (x < 2), 4 / x**2, 0)
    bound = np.sum(w * (16 + lost + 40), axis=1) * 2.0**-53
    assert np.all(np.abs(got - ref) <= bound), float(np.max(np.abs(got - ref) / bound))
