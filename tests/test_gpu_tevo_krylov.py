"""The Chebyshev evaluation of <e1|exp(-i s (T - e0) t)|e1> against dense 64-bit eigenpairs, at the
edges of its blocks, for both signs, at zero, tiny, negative and long times, and the hand-over to
the eigenpairs of T beyond the expansion's largest order."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(m, seed):
    r = np.random.default_rng(seed)
    a = r.uniform(-8, 8, m)
    b = np.concatenate([[3.0], r.uniform(0.5, 4, m - 1), [1e-3]])
    return a, b


def _reference(a, b, norm2, e0, sign, t):
    m = len(a)
    lam, U = np.linalg.eigh(np.diag(a) + np.diag(b[1:m], 1) + np.diag(b[1:m], -1))
    return -1j * sign * norm2 * (np.exp(-1j * sign * np.outer(t, lam - e0)) @ U[0] ** 2)


@pytest.mark.parametrize("m", [1, 2, 3, 32, 511, 512, 513, 1100, 4096])
@pytest.mark.parametrize("sign,t_max", [(1, 20.0), (-1, 3.0)])
def test_against_eigenpairs(cuda, m, sign, t_max):
    from cmpy_gb300 import engine as E

    a, b = _case(m, m)
    t = np.concatenate([[0.0, 1e-14, -1e-11, 1e-7, -t_max / 3], np.linspace(0, t_max, 60)])
    e0, norm2 = -3.7, 0.61
    got = E.tevo_krylov(a, b, norm2, e0, sign, t).cpu().numpy()
    ref = _reference(a, b, norm2, e0, sign, t)
    # one rounding a step of the recurrence and of the phases on both sides; |T| <= 16
    tol = 16 * (16 * t_max + 14 * (16 * t_max) ** (1 / 3) + 64) * 2.0**-53 * norm2
    assert np.max(np.abs(got - ref)) <= tol


@pytest.mark.parametrize("m", [5, 300])
def test_long_times_take_the_eigenpairs(cuda, m):
    from cmpy_gb300 import engine as E

    a, b = _case(m, 7)
    t = np.array([0.0, 10.0, 4e4])
    got = E.tevo_krylov(a, b, 1.0, 0.3, 1, t).cpu().numpy()
    assert np.max(np.abs(got - _reference(a, b, 1.0, 0.3, 1, t))) <= 16 * 16 * 4e4 * 2.0**-53


def test_split_chain_and_non_finite(cuda):
    """A zero coupling inside T (an exhausted Krylov space), and NaN coefficients."""
    from cmpy_gb300 import engine as E

    a, b = _case(40, 9)
    b[17] = 0.0
    t = np.linspace(0, 5, 33)
    got = E.tevo_krylov(a, b, 1.0, 0.0, 1, t).cpu().numpy()
    assert np.max(np.abs(got - _reference(a, b, 1.0, 0.0, 1, t))) <= 16 * 220 * 2.0**-53
    g0 = E.tevo_krylov(np.full(6, 2.5), np.zeros(7), 1.0, 0.0, 1, t).cpu().numpy()
    assert np.max(np.abs(g0 + 1j * np.exp(-2.5j * t))) <= 16 * 64 * 2.0**-53
