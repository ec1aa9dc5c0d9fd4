"""compute_groundstate with its small sectors in one launch against sector after sector: converged and
cut-off runs (the same start vectors, so the same coefficients), two CTAs to an SM and one, clusters
of 8, 4 and 2, a model of one large sector's neighbours. Energies to 1e-12 of |H|: the coefficients
agree bit for bit, the tridiagonal solvers round differently."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(n, kind):
    from cmpy_gb300.models import HubbardModel

    nb = [(i, i + 1) for i in range(n - 1)]
    if kind == "chain":
        return HubbardModel(n, nb, inter=4.0, eps=0.0, hop=1.0, mu=2.0)
    r = np.random.default_rng(n)
    return HubbardModel(n, nb, inter=r.uniform(1, 4, n), eps=r.uniform(-1, 1, n), hop=0.5, mu=0.3)


@pytest.mark.parametrize("n,kind,steps", [(3, "chain", 400), (5, "disorder", 400), (6, "chain", 400), (6, "disorder", 7),
                                          (8, "chain", 60), (8, "disorder", 400), (9, "disorder", 40)])
def test_same_as_sector_by_sector(cuda, n, kind, steps):
    from cmpy_gb300 import exactdiag as X

    m = _model(n, kind)
    fillings = list(m.basis.iter_fillings())
    ref = {f: X.groundstate_sector(m, *f, max_steps=steps)[0] for f in fillings}
    scale = max(abs(e) for e in ref.values())
    got = X._resident_energies(m, fillings, steps, 1e-12)
    assert len(got) > 1
    for f, (e, v) in got.items():
        assert v is None
        if m.plan(*f).dim > 50:
            assert abs(e - ref[f]) <= 1e-12 * scale, f
    gs = X.compute_groundstate(m, max_steps=steps)
    e0 = min(ref.values())
    assert abs(gs.energy - e0) <= 1e-12 * scale
    assert abs(ref[gs.n_up, gs.n_dn] - e0) <= 1e-12 * scale
    h = m.plan(gs.n_up, gs.n_dn)
    psi = torch.as_tensor(gs.state).cuda()
    assert psi.numel() == h.dim and abs(float(psi.norm()) - 1) < 1e-12
    if steps == 400:
        assert float((h.matvec(psi) - gs.energy * psi).norm()) < 1e-9 * scale
