"""Real-time G with only as many Lanczos levels as it can depend on, against all levels asked for:
short and long times, both directions, negative times, both kinds of sectors; the interval that fixes the
number against the spectrum. 1e-12: both are sums of Chebyshev terms rounded at 1e-16 each, up to
1e3 of them."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(n, seed):
    from cmpy_gb300.models import HubbardModel

    nb = [(i, i + 1) for i in range(n - 1)]
    if seed == 0:
        return HubbardModel(n, nb, inter=4.0, eps=0.0, hop=1.0, mu=2.0)
    r = np.random.default_rng(seed)
    return HubbardModel(n, nb, inter=r.uniform(-2, 4, n), eps=r.uniform(-1, 1, n), hop=0.7, mu=0.3)


@pytest.mark.parametrize("n,seed", [(2, 0), (5, 1), (6, 0), (7, 2), (8, 0)])
@pytest.mark.parametrize("t0,t1", [(0.0, 0.0), (0.0, 0.1), (-3.0, 20.0), (0.0, 60.0)])
def test_same_as_all_levels(cuda, monkeypatch, n, seed, t0, t1):
    from cmpy_gb300 import exactdiag as X

    m = _model(n, seed)
    gs = X.compute_groundstate(m)
    for f in (X.gf_greater, X.gf_lesser):
        t, g = f(m, gs, t0, t1, 50)
        with monkeypatch.context() as c:
            c.setattr(X, "_tevo_levels", lambda plan, times: 4096)
            _, ref = f(m, gs, t0, t1, 50)
        assert np.max(np.abs(g - ref)) < 1e-12


@pytest.mark.parametrize("n,seed", [(3, 1), (4, 0), (5, 3)])
def test_spectrum_bounds(cuda, n, seed):
    m = _model(n, seed)
    for f in m.basis.iter_fillings():
        p = m.plan(*f)
        w = np.linalg.eigvalsh(p.dense().cpu().numpy())
        lo, hi = p.spectrum_bounds()
        assert lo <= w[0] + 1e-12 and w[-1] <= hi + 1e-12


def test_refused_sizes_stay_refused(cuda):
    from cmpy_gb300 import exactdiag as X

    m = _model(9, 0)
    psi = np.zeros(m.plan(4, 4).dim)
    psi[0] = 1.0
    gs = X.EigenState(-1.0, psi, 4, 4)
    with pytest.raises(ValueError):  # the sector has more than 4096 states
        X.gf_greater(m, gs, 0.0, 1.0, 5, n_lev=None)
