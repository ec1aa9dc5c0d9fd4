"""The clusters that compute_groundstate runs its small sectors on hold the vectors of the largest one."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 8, 9, 10])
def test_vectors_fit(cuda, monkeypatch, n):
    from cmpy_gb300 import exactdiag as X
    from cmpy_gb300.batched import Batch
    from cmpy_gb300.models import HubbardModel

    r = np.random.default_rng(n)
    m = HubbardModel(n, [(i, i + 1) for i in range(n - 1)], inter=r.uniform(1, 4, n), eps=r.uniform(-1, 1, n), hop=0.5)
    seen, plain = [], Batch.lanczos

    def spy(self, *args, **kw):
        seen.append((max(self.dims), self.ctas_per_sm, self.cluster_size))
        return plain(self, *args, **kw)

    monkeypatch.setattr(Batch, "lanczos", spy)
    got = X._resident_energies(m, list(m.basis.iter_fillings()), 200, 1e-12)
    ((dmax, per_sm, cluster),) = seen
    # a copy of R, and the CTA's share of W and R_{k-1}, in an SM's 228 KB
    assert (8 + 16 / cluster) * dmax * per_sm <= 228 * 1024
    f = max(got, key=lambda q: m.plan(*q).dim)
    e = X.groundstate_sector(m, *f, max_steps=200)[0]
    assert abs(got[f][0] - e) <= 1e-12 * max(1.0, abs(e))
