"""The Lehmann pole sum split over blocks: sizes at the edges of its tiles and chunks against a
64-bit numpy sum of the same poles, and the reciprocal at the ends of its range."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(e, ep, ov, beta, emin, z):
    w = np.exp(-beta * (e - emin)) if np.isfinite(beta) else np.ones_like(e)
    wp = np.exp(-beta * (ep - emin)) if np.isfinite(beta) else np.ones_like(ep)
    c = ov * (w[None, :] + wp[:, None])
    p = ep[:, None] - e[None, :]
    return np.array([np.sum(c / (zz - p)) for zz in z]), np.array([np.sum(np.abs(c / (zz - p))) for zz in z])


@pytest.mark.parametrize("nd,ndp,nz", [(1, 1, 1), (3, 5, 7), (16, 16, 128), (17, 15, 129), (64, 37, 255),
                                       (300, 400, 512), (1, 2000, 3), (257, 1, 1000)])
@pytest.mark.parametrize("beta", [4.0, float("inf")])
def test_split_sum(cuda, nd, ndp, nz, beta):
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(nd * 1000 + ndp)
    e, ep = np.sort(r.uniform(-6, 6, nd)), np.sort(r.uniform(-6, 6, ndp))
    ov = r.uniform(0, 1, (ndp, nd)) ** 2
    ov[r.random((ndp, nd)) < 0.3] = 0.0
    z = np.linspace(-9, 9, nz) + 0.03j
    ref, mag = _reference(e, ep, ov, beta, e[0], z)
    g = torch.full((nz,), 0.25 - 0.5j, dtype=torch.complex128, device="cuda")
    E.lehmann_accumulate(e, ep, ov, beta, float(e[0]), z, g)
    # every term is off by a few roundings of the pole difference (|p| <= 12, |z - p| >= 0.03: its
    # relative error is up to 12 / 0.03 * 2^-53) and the sum by at most nd * ndp roundings
    tol = (12 / 0.03 + 16 + nd * ndp) * 2.0**-53
    err = np.abs(g.cpu().numpy() - (0.25 - 0.5j) - ref)
    assert np.all(err <= tol * mag + 2.0**-52), float(np.max(err / np.maximum(mag, 1e-300)))


@pytest.mark.parametrize("eta", [1e-160, 1e-150, 1e-3, 1.0, 1e150, 1e160])
def test_reciprocal_range(cuda, eta):
    """One pole seen from distances whose squares leave the range of the fast reciprocal (or the
    doubles): as the plain division."""
    from cmpy_gb300 import engine as E

    g = torch.zeros(1, dtype=torch.complex128, device="cuda")
    E.lehmann_accumulate([0.0], [0.0], [[0.5]], float("inf"), 0.0, np.array([1j * eta]), g)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore", under="ignore"):
        den = np.float64(eta) * np.float64(eta)
        want = -np.float64(eta) * (np.float64(1.0) / den)
    got = g.cpu().numpy()[0].imag
    assert (np.isnan(want) and np.isnan(got)) or got == want or abs(got - want) <= 4 * 2.0**-53 * abs(want)
