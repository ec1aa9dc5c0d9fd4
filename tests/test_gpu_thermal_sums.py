"""The one-pass thermal sums against the tensor expressions: both species, both layouts of the
eigenvectors and a strided one, sectors of one state to a few blocks, a lower and a higher running
energy. 1e-13 relative: sums of positive terms in FP64."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,a,b", [(1, 0, 0), (1, 1, 1), (3, 1, 2), (6, 3, 2), (6, 3, 3), (7, 3, 4)])
@pytest.mark.parametrize("layout", ["rows", "columns", "strided"])
@pytest.mark.parametrize("beta,emin", [(3.0, np.inf), (50.0, -1e3), (0.0, 5.0)])
def test_sums(cuda, n, a, b, layout, beta, emin):
    from cmpy_gb300 import engine as E
    from cmpy_gb300.basis import Basis
    from cmpy_gb300 import exactdiag as X

    sec = Basis(n).get_sector(a, b)
    D = len(sec.up_states) * len(sec.dn_states)
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.sort(torch.randn(D, generator=g, device="cuda", dtype=torch.float64)).values
    v = torch.randn(D, D, generator=g, device="cuda", dtype=torch.float64)
    if layout == "columns":
        v = v.t()
    elif layout == "strided":
        v = torch.randn(D, 3 * D, generator=g, device="cuda", dtype=torch.float64)[:, ::3]
    e0 = min(emin, float(w.min()))
    for site in range(n):
        for sigma in (1, 2):
            m, z, occ, dbl = E.thermal_sums(w, v, sec.up_states, sec.dn_states, site, sigma == 2, beta, emin)
            assert m == float(w.min())
            zr = float(torch.exp(-beta * (w - e0)).sum())
            assert abs(z - zr) <= 1e-13 * zr
            r = X.occupation(sec.up_states, sec.dn_states, w, v, beta, e0, site, sigma)
            assert abs(occ - r) <= 1e-13 * abs(r)
            r = X.double_occupation(sec.up_states, sec.dn_states, w, v, beta, e0, site)
            assert abs(dbl - r) <= 1e-13 * abs(r)
    m, z, occ, dbl = E.thermal_sums(w, v, sec.up_states, sec.dn_states, 0, False, beta, emin, occ=False)
    assert abs(z - zr) <= 1e-13 * zr and occ == 0.0 and dbl == 0.0
    with pytest.raises(ValueError):
        E.thermal_sums(w, v[:, : D - 1] if D > 1 else v[:0], sec.up_states, sec.dn_states, 0, False, beta, emin)
