"""The pole sum's reciprocal over mantissas and exponents: one pole on the real axis, G(z) = 1 / (z - pole) formed as
(z - pole) * rcp((z - pole)^2), against extended precision."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _error(x):
    """Relative error of the device's x * rcp(fl(x^2)), in units of 2^-53."""
    from cmpy_gb300 import engine as E

    g = torch.zeros(len(x), dtype=torch.complex128, device="cuda")
    E.lehmann_accumulate([0.0], [0.0], [[0.5]], float("inf"), 0.0, x.astype(complex), g)
    got = g.cpu().numpy().real.astype(np.longdouble)
    want = x.astype(np.longdouble) / (x * x).astype(np.longdouble)
    return float(np.max(np.abs(got - want) / np.abs(want)) * np.longdouble(2) ** 53)


def test_mantissas(cuda):
    # both binades of x^2, evenly and around the ends
    x = np.concatenate([1 + np.arange(1 << 19) / 2.0**19, 1 + np.arange(64) * 2.0**-52, 2 - np.arange(1, 65) * 2.0**-52,
                        np.sqrt(2.0) * (1 + np.arange(-64, 64) * 2.0**-52),
                        np.random.default_rng(0).uniform(1, 2, 1 << 19)])
    # one rounding of the product, one of the step, and 2^-7 of one for what the step leaves out
    assert _error(x) <= 2 + 2.0**-6


@pytest.mark.parametrize("power", [-499, -300, -40, 60, 300, 499])
def test_exponents(cuda, power):
    x = np.random.default_rng(abs(power)).uniform(1, 2, 4096) * 2.0**power
    assert _error(np.concatenate([x, -x])) <= 2 + 2.0**-6
