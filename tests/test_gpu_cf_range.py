"""The continued fraction at the ends of the doubles' range: parameters in units that are powers of two (every
operation scales exactly, so the value does) and frequencies far outside the spectrum."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(n):
    r = np.random.default_rng(n)
    a = r.uniform(-8, 8, n)
    b = np.concatenate([[0.0], r.uniform(0.2, 4, n)])
    z = np.concatenate([np.linspace(-12, 12, 67) + 0.05j, 1j * np.array([1e-3, 0.3, 50.0])])
    return a, b, z


@pytest.mark.parametrize("n", [1, 2, 200, 600])
@pytest.mark.parametrize("power", [-480, -400, -330, -200, 200, 330, 400, 500])
def test_units(cuda, n, power):
    from cmpy_gb300 import engine as E
    from cmpy_gb300.batched import BatchResult, batch_cf

    a, b, z = _problem(n)
    s = 2.0**power
    ref = E.continued_fraction(a, b, 0.7, z, e0=-1.25).cpu().numpy()
    got = E.continued_fraction(s * a, s * b, 0.7, s * z, e0=-1.25 * s).cpu().numpy()
    assert np.all(np.isfinite(ref)) and np.array_equal(got, ref / s)
    t = lambda x: torch.as_tensor(np.asarray(x)).cuda()
    b[0] = 1.0  # (the norm)
    res = lambda f: BatchResult(None, t(np.array([n], np.int32)), None, t(f * a[None]),
                                t(np.concatenate([[1.0], f * b[1:]])[None]), None)
    one = batch_cf(res(1.0), t([-1.25]), 1, z).cpu().numpy()
    assert np.array_equal(batch_cf(res(s), t([-1.25 * s]), 1, s * z).cpu().numpy(), one / s)


@pytest.mark.parametrize("n", [1, 2, 200, 600])
def test_far_frequencies(cuda, n):
    """G(z) = norm / z up to the rounding of z - a and the quotient's (four operations)."""
    from cmpy_gb300 import engine as E

    a, b, _ = _problem(n)
    z = np.array([m * np.exp(1j * f) for m in (1e20, 1e90, 1e97, 1e100, 1e120, 1e150) for f in (0.1, 1.3, 3.0)])
    got = E.continued_fraction(a, b, 0.7, z).cpu().numpy()
    assert np.all(np.abs(got * z - 0.7) <= 16 * 2.0**-53 + 8.0 / np.abs(z))
