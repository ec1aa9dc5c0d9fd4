"""The continued fraction's error against extended precision is that of the tails t_l = z - a_l - b_{l+1}^2 / t_{l+1}
in doubles: their ratio over many sets of coefficients, on the Matsubara axis and near the real one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fma(x, y, z):
    return (x.astype(np.longdouble) * y + z).astype(float)


def _tails(a, b, z):
    tr, tm = z.real - a[-1], z.imag
    for k in range(len(a) - 2, -1, -1):
        inv = b[k + 1] ** 2 / _fma(tr, tr, tm * tm)
        tr, tm = _fma(-tr, inv, z.real - a[k]), _fma(tm, inv, z.imag)
    inv = 1.0 / _fma(tr, tr, tm * tm)
    return tr * inv - 1j * (tm * inv)


def _extended(a, b, z):
    z, a, b = z.astype(np.clongdouble), a.astype(np.longdouble), b.astype(np.longdouble)
    t = z - a[-1]
    for k in range(len(a) - 2, -1, -1):
        t = z - a[k] - b[k + 1] ** 2 / t
    return 1 / t


@pytest.mark.parametrize("eta", [None, 0.05, 0.2])
def test_error_of_the_tails(cuda, eta):
    from cmpy_gb300 import engine as E

    ratio = []
    for seed in range(400):
        r = np.random.default_rng(seed)
        n = int(r.integers(10, 250))
        if seed % 2:
            a, b = r.uniform(-8, 8, n), r.uniform(0.2, 4, n + 1)
        else:
            a, b = r.normal(0, 0.5) + 0.3 * r.standard_normal(n), 2.5 + 0.4 * r.standard_normal(n + 1)
        b[0] = 0.0
        z = 1j * (2 * np.arange(64) + 1) * np.pi / 30 if eta is None else np.linspace(-12, 12, 64) + 1j * eta
        ref = _extended(a, b, z)
        rms = lambda g: float(np.sqrt(np.mean(np.abs(g - ref) ** 2)))
        ratio.append(rms(E.continued_fraction(a, b, 1.0, z).cpu().numpy()) / rms(_tails(a, b, z)))
    # (a set's ratio scatters by 0.3 to 0.6 about one; 400 of them average to 0.015 to 0.03)
    assert np.exp(np.mean(np.log(ratio))) <= 1.04
