"""The Laplace transform of sampled G(t) with its segments split over blocks."""

import numpy as np
import pytest

from oracle import ed_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,nz", [(1, 5), (2, 1), (3, 127), (10, 129), (1217, 128), (2500, 3), (333, 1500)])
@pytest.mark.parametrize("method", ["lin", "trapz"])
def test_laplace_split_sizes(cuda, nt, nz, method):
    """Segments split over blocks: chunk and tile edges, non-uniform times, both branches of the
    segment weights, against a 64-bit numpy sum."""
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(nt * 7 + nz)
    t = np.cumsum(r.uniform(0.01, 0.2, nt))
    g = r.standard_normal(nt) + 1j * r.standard_normal(nt)
    z = np.linspace(-6, 6, nz) + 0.05j
    got = E.laplace_t2z(t, g, z, method=method).cpu().numpy()
    if method == "lin":
        ref = O.laplace_lin(t, g, z) if nt > 1 else np.zeros(nz, complex)
    else:
        f = np.exp(1j * z[:, None] * t[None, :]) * g[None, :]
        ref = 0.5 * np.sum((f[:, 1:] + f[:, :-1]) * np.diff(t)[None, :], axis=1)
    # per segment: the phase u t (up to |u| t_last) carries its argument's rounding, the weights
    # near |u h| = 1/4 lose up to 4^2 of a cancellation; the magnitudes add up to sum h |g|
    mag = np.sum(np.diff(t) * (np.abs(g[1:]) + np.abs(g[:-1]))) if nt > 1 else 0.0
    tol = (6.1 * (t[-1] + 1) + 64 + nt) * 2.0**-52
    assert np.max(np.abs(got - ref)) <= tol * mag
