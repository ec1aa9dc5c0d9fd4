"""A small sector's Lanczos run in one launch against the launched steps (forced by naming a matvec
kernel): sectors from one state to the largest that fits a cluster and the first that does not."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SECTORS = [(1, 0, 0, "u"), (2, 1, 1, "u"), (3, 3, 1, "u"), (5, 2, 3, "d"), (6, 3, 3, "u"), (7, 3, 4, "d"),
           (8, 4, 4, "u"), (9, 4, 4, "d"), (9, 4, 5, "u"), (10, 4, 4, "u")]


def _plan(n, a, b, kind):
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(n)
    hop = [(i, i + 1, 1.0 if kind == "u" else -0.5) for i in range(n - 1)]
    if kind == "u":
        return E.Plan.fermion(n, [-2.0] * n, [4.0] * n, hop, a, b)
    return E.Plan.fermion(n, r.uniform(-1, 1, n), r.uniform(1, 4, n), hop, a, b)


def _launched(plan):
    plan.set_matvec_variant(1)
    return plan


def _start(plan, seed=1):
    return torch.as_tensor(np.random.default_rng(seed).uniform(0.1, 1, plan.dim)).cuda()


@pytest.mark.parametrize("sec", SECTORS)
def test_coefficients(cuda, sec):
    """The first 12 coefficients to the growth of their rounding (1e-10 of |H| < 64); one matvec is
    exact in both, the sums and scalars are FP64."""
    from cmpy_gb300 import engine as E

    p, q = _plan(*sec), _launched(_plan(*sec))
    v = _start(p)
    a, b, nrm = E.lanczos_coeffs(p, v, 12)
    ar, br, nr = E.lanczos_coeffs(q, v, 12)
    m = min(a.numel(), ar.numel())
    assert a.numel() == ar.numel() or (p.dim < 12 and float(br[m].abs()) < 1e-10)
    assert abs(nrm - nr) <= 1e-14 * nr and float(b[0]) == 0.0
    k = max(1, m - 1) if p.dim < 12 else m
    assert float((a[:k] - ar[:k]).abs().max()) < 1e-10
    assert float((b[:k] - br[:k]).abs().max()) < 1e-10
    # two runs in one call: the same bits as separate ones
    w = _start(p, 2)
    one = E.lanczos_coeffs(p, w, 12)
    for x, y in zip(E.lanczos_coeffs_multi([(p, v), (p, w)], 12), ((a, b, nrm), one)):
        assert torch.equal(x[0], y[0]) and torch.equal(x[1], y[1]) and x[2] == y[2]


@pytest.mark.parametrize("sec", SECTORS)
@pytest.mark.parametrize("tol,check", [(1e-12, 10), (1e-10, 1), (0.0, 0)])
def test_groundstate(cuda, sec, tol, check):
    """Energy to 1e-11 and the vector's true residual to what the run reports plus rounding."""
    from cmpy_gb300 import engine as E

    p, q = _plan(*sec), _launched(_plan(*sec))
    K = 200 if p.dim <= 20000 else 120
    v = _start(p)
    r = E.lanczos(p, max_steps=K, tol=tol, check_every=check, v0=v)
    ref = E.lanczos(q, max_steps=K, tol=tol, check_every=check, v0=v)
    assert abs(r.energy - ref.energy) < 1e-11 * max(1.0, abs(ref.energy))
    assert r.converged == ref.converged or p.dim < K
    if tol > 0 and p.dim > K:
        assert abs(r.steps - ref.steps) <= 2 * check
    assert abs(float(r.vector.norm()) - 1.0) < 1e-13
    h = p.matvec(r.vector)
    assert np.isnan(r.residual) == np.isnan(ref.residual)  # (of a zero matrix)
    assert float((h - r.energy * r.vector).norm()) < 2 * np.nan_to_num(r.residual) + 1e-9
    n = E.lanczos(p, max_steps=K, tol=tol, check_every=check, v0=v, want_vector=False)
    assert n.energy == r.energy and n.steps == r.steps and torch.equal(n.alpha, r.alpha)


def test_starts_and_streams(cuda):
    from cmpy_gb300 import engine as E

    p = _plan(6, 3, 2, "u")
    z = torch.zeros(p.dim, dtype=torch.float64, device="cuda")
    bad = z.clone()
    bad[7] = float("nan")
    a, b, n = E.lanczos_coeffs(p, z, 20)
    assert a.numel() == 0 and n == 0.0
    with pytest.raises(Exception):
        E.lanczos_coeffs(p, bad, 20)
    for v in (z, bad):
        with pytest.raises(Exception):
            E.lanczos(p, max_steps=20, v0=v)
    ref = E.lanczos(p, max_steps=60, tol=1e-12, check_every=10, seed=3)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        r = E.lanczos(p, max_steps=60, tol=1e-12, check_every=10, seed=3)
    s.synchronize()
    assert r.energy == ref.energy and torch.equal(r.vector, ref.vector)
    # per-matvec times still come from launched steps
    assert E.lanczos(p, max_steps=20, profile=True).matvecs == 20
