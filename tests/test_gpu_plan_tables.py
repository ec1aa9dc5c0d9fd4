"""Sector tables built on the host (up to 8192 states per spin; a state index by table up to 16
sites, by binary search above) and by kernels (more states): H x against the oracle's triplets, and
the variants whose tables are built when they are asked for."""

import numpy as np
import pytest
import torch

from oracle import ed_oracle as O

pytestmark = pytest.mark.gpu


def _ring(n):
    return [(i, i + 1, 1.0) for i in range(n - 1)] + [(0, n - 1, 1.0)]


@pytest.mark.parametrize("n,nu,nd,hop", [(1, 0, 1, 1.0), (2, 1, 1, 1.0), (5, 0, 5, 1.0), (9, 4, 3, 0.7), (16, 2, 1, 1.0),
                                         (17, 3, 1, 0.7), (18, 2, 2, 1.0), (16, 5, 1, 1.0), (16, 7, 1, 0.7),
                                         (16, 1, 7, 1.0), (16, 8, 0, 1.0)])
def test_matvec_against_triplets(cuda, n, nu, nd, hop):
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(n * 100 + nu)
    eps, u = r.uniform(-1, 1, n), r.uniform(0, 4, n)
    bonds = [(i, j, hop) for i, j, _ in _ring(n)] if n > 2 else ([(0, 1, hop)] if n == 2 else [])
    p = E.Plan.fermion(n, eps, u, bonds, nu, nd)
    up, dn = O.sector_states(n, nu), O.sector_states(n, nd)
    rows, cols, vals = O.coo_fermion(up, dn, eps, u, bonds, n)
    x = r.standard_normal(p.dim)
    y = p.matvec(torch.as_tensor(x).cuda()).cpu().numpy()
    ref = np.bincount(cols, weights=vals * x[rows], minlength=p.dim)
    mag = np.bincount(cols, weights=np.abs(vals * x[rows]), minlength=p.dim)
    # at most 2 n + 4 terms a row, each with a product and a sum on either side
    assert np.all(np.abs(y - ref) <= (2 * n + 4) * 2.0**-52 * mag + 1e-300)
    h = np.abs(np.bincount(cols, weights=np.abs(vals), minlength=p.dim))
    assert p.hnorm_bound >= h.max() * (1 - 1e-14)


@pytest.mark.parametrize("nu,nd", [(3, 3), (4, 2)])
def test_two_pass_tables_on_request(cuda, nu, nd):
    from cmpy_gb300 import engine as E

    p = E.Plan.fermion(8, [-2.0] * 8, [4.0] * 8, _ring(8), nu, nd)
    x = torch.randint(-(2**40), 2**40, (p.dim,), dtype=torch.int64, device="cuda")
    ref, e = p.matvec_fixed(x, 0)
    assert p.matvec_variant == 7
    for v in (5, 6, 3, 5, 0):
        p.set_matvec_variant(v)
        assert p.matvec_variant == (v or 7)
        y, e2 = p.matvec_fixed(x, 0)
        assert e2 == e and torch.equal(y, ref)
