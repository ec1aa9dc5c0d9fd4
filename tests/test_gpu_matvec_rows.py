"""The FP64 matvec by rows against the dense matrix: one hopping and many, uniform diagonals and others,
sectors of one state to several blocks' widths, vectors and blocks of vectors."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _models():
    r = np.random.default_rng(5)
    yield "chain", lambda n: ([-1.3] * n, [2.6] * n, [(i, i + 1, 0.7) for i in range(n - 1)], None)
    yield "ring", lambda n: ([0.1] * n, list(r.uniform(0, 4, n)), [(i, i + 1, 1.0) for i in range(n - 1)] + [(0, n - 1, 1.0)], n)
    yield "star", lambda n: (list(r.uniform(-2, 2, n)), [3.3] + [0.0] * (n - 1),
                             [(0, i, float(v)) for i, v in enumerate(r.uniform(-0.6, 0.6, n - 1), 1)], n)
    yield "levels", lambda n: (list(r.uniform(-2, 2, n)), [1.7] * n, [(i, i + 1, -0.3) for i in range(n - 1)], None)
    yield "zero", lambda n: ([0.0] * n, [1.1] * n, [(0, 1, 0.0), (1, 2, 0.5)], None)
    yield "no hops", lambda n: ([0.2] * n, [0.3] * n, [], None)


@pytest.mark.parametrize("sector", [(3, 1, 1), (3, 0, 2), (3, 3, 3), (4, 2, 0), (6, 3, 2), (9, 1, 4), (9, 4, 3), (11, 2, 5), (13, 1, 6)])
@pytest.mark.parametrize("which", range(6))
def test_against_dense(cuda, which, sector):
    from cmpy_gb300 import engine as E

    _, make = list(_models())[which]
    n, nu, nd = sector
    eps, u, bonds, width = make(n)
    p = E.Plan.fermion(n, eps, u, bonds, nu, nd, **({} if width is None else {"sign_width": width}))
    H = p.dense()
    X = torch.randn(p.dim, 3, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    # each side rounds once a term of the row and of the diagonal's own sum, whose terms may cancel
    terms = int((H != 0).sum(1).max()) + 2 * n + 2
    diag = 2 * sum(map(abs, eps)) + sum(map(abs, u))
    limit = 2 * terms * 2.0**-53 * (H.abs() @ X.abs() + diag * X.abs()) + 1e-300
    assert bool(((p.matmat(X) - H @ X).abs() <= limit).all())
    # (a single vector of a small sector takes the other FP64 kernel: the same operations in the same order)
    assert torch.equal(p.matmat(X)[:, 1], p.matvec(X[:, 1].contiguous()))
    many = X[:, :1].expand(-1, max(1, -(-16384 // p.dim))).contiguous()
    assert bool((p.matmat(many) == p.matvec(many[:, 0].contiguous())[:, None]).all())
