"""A model that makes its sectors' plans itself is solved with them, also where many sectors go into one launch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _models(n=5):
    from cmpy_gb300 import engine as E
    from cmpy_gb300.models import HubbardModel

    bonds = [(i, i + 1) for i in range(n - 1)]

    class Shifted(HubbardModel):
        """The Hubbard chain with its levels moved in the plans alone."""

        def plan(self, n_up, n_dn):
            eps, u, hops, width = self.fermion_descriptor()
            return E.Plan.fermion(n, np.asarray(eps) + 0.375, u, hops, n_up, n_dn, width)

    class Same(HubbardModel):
        def plan(self, n_up, n_dn):
            return super().plan(n_up, n_dn)

    kw = dict(inter=4.0, hop=1.0, mu=2.0)
    return Shifted(n, bonds, eps=0.0, **kw), HubbardModel(n, bonds, eps=0.375, **kw), Same(n, bonds, eps=0.375, **kw)


def test_own_plans_are_used(cuda):
    from cmpy_gb300 import batched as B
    from cmpy_gb300 import exactdiag as X

    own, ref, same = _models()
    z = np.linspace(-3, 3, 9) + 0.2j
    for m in (own, same):
        a, b = X.compute_groundstate(m), X.compute_groundstate(ref)
        assert (a.n_up, a.n_dn) == (b.n_up, b.n_dn) and abs(a.energy - b.energy) < 1e-11
        assert np.allclose(X.gf_lehmann(m, z, 5.0).gf, X.gf_lehmann(ref, z, 5.0).gf, rtol=0, atol=1e-10)
        e = [B.groundstate_all_sectors(q)[1].energy.cpu().numpy() for q in (m, ref)]
        assert np.abs(e[0] - e[1]).max() < 1e-11
    assert own.plans([None, (2, 2)])[0] is None
