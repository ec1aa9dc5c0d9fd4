"""The batched Lanczos kernel with its vectors in shared memory: every launch configuration (one CTA
of 288, 544 and 800 threads, clusters of 2, 4 and 8), sectors from one state to more than a CTA's
shared memory holds, both diagonals, site-dependent U, odd sector lengths."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ONE = [(128, 4, 1), (256, 2, 1), (256, 3, 1), (512, 1, 1), (512, 2, 1), (1024, 1, 1)]
CLUSTER = [(512, 2, 2), (1024, 1, 2), (512, 2, 4), (1024, 1, 4), (512, 2, 8), (1024, 1, 8)]


def _plans(which):
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(11)
    ring = lambda n: [(i, i + 1, 1.0) for i in range(n - 1)] + ([(0, n - 1, 1.0)] if n > 2 else [])
    chain = lambda n: [(i, i + 1, -0.5) for i in range(n - 1)]
    if which == "small":
        sec = [(3, 0, 0), (3, 3, 1), (4, 2, 2), (5, 2, 1), (6, 3, 3), (6, 2, 3), (7, 3, 4), (8, 4, 4)]
        return [E.Plan.fermion(n, [-1.5] * n, [3.0] * n, ring(n), a, b) for n, a, b in sec]
    if which == "disorder":
        sec = [(5, 2, 3), (6, 1, 4), (7, 4, 3), (8, 3, 2), (8, 4, 4)]
        return [E.Plan.fermion(n, r.uniform(-1, 1, n), r.uniform(1, 4, n), chain(n), a, b) for n, a, b in sec]
    return [E.Plan.fermion(10, [-2.0] * 10, [4.0] * 10, ring(10), 5, 5),
            E.Plan.fermion(9, [-2.0] * 9, [4.0] * 9, chain(9), 4, 5)]


def _run(plans, cfg, K, vectors=False):
    from cmpy_gb300.batched import Batch

    b = Batch(plans)
    b.threads, b.ctas_per_sm, b.cluster_size = cfg
    starts = [torch.as_tensor(np.random.default_rng(i).uniform(0.1, 1, p.dim)).cuda() for i, p in enumerate(plans)]
    r = b.lanczos(max_steps=K, tol=0.0, check_every=0, starts=starts, want_vector=vectors)
    a, be, st = b.coeffs(K, starts)
    torch.cuda.synchronize()
    assert torch.equal(st, r.steps)
    for i, m in enumerate(st.tolist()):
        assert torch.equal(a[i, :m], r.alpha[i, :m]) and torch.equal(be[i, :m + 1], r.beta[i, :m + 1])
    return r


@pytest.mark.parametrize("which,K", [("small", 30), ("disorder", 30), ("large", 12)])
def test_configurations_agree(cuda, which, K):
    from cmpy_gb300 import engine as E

    plans = _plans(which)
    ref = _run(plans, ONE[1], K, vectors=which != "large")
    for cfg in ONE[2:] + ONE[:1]:  # one order of the sums: the same bits
        r = _run(plans, cfg, K, vectors=which != "large")
        assert torch.equal(r.steps, ref.steps) and torch.equal(r.energy, ref.energy)
        for i, m in enumerate(ref.steps.tolist()):
            assert torch.equal(r.alpha[i, :m], ref.alpha[i, :m]) and torch.equal(r.beta[i, :m + 1], ref.beta[i, :m + 1])
            if r.vectors is not None:
                assert torch.equal(r.vectors[i], ref.vectors[i])
    for cfg in CLUSTER:  # exact sums: the first steps to rounding (it grows along the recurrence)
        r = _run(plans, cfg, K)
        for i, m in enumerate(ref.steps.tolist()):
            k = min(m, 8)
            assert torch.allclose(r.alpha[i, :k], ref.alpha[i, :k], rtol=0, atol=1e-11)
            assert torch.allclose(r.beta[i, :k], ref.beta[i, :k], rtol=1e-11, atol=1e-11)
    for i, p in enumerate(plans):  # the launch-per-step runs
        start = torch.as_tensor(np.random.default_rng(i).uniform(0.1, 1, p.dim)).cuda()
        a, b, nrm = E.lanczos_coeffs(p, start, max_steps=K)
        k = min(int(ref.steps[i]), a.numel(), 8)
        assert torch.allclose(ref.alpha[i, :k], a[:k], rtol=0, atol=1e-11)
        assert abs(float(ref.beta[i, 0]) - nrm) <= 1e-13 * nrm


@pytest.mark.parametrize("cfg", [ONE[2], ONE[4], ONE[5], CLUSTER[0], CLUSTER[5]])
def test_ground_states_against_dense(cuda, cfg):
    from cmpy_gb300.batched import Batch

    plans = _plans("small") + _plans("disorder")[:3]
    b = Batch(plans)
    b.threads, b.ctas_per_sm, b.cluster_size = cfg
    r = b.lanczos(max_steps=300, tol=1e-12, check_every=10, want_vector=True)
    for i, p in enumerate(plans):
        if p.dim > 1300:
            continue
        h = p.dense()
        w = torch.linalg.eigvalsh(h)
        e = float(r.energy[i])
        assert abs(e - float(w[0])) <= 1e-10 * max(1.0, abs(float(w[0])))
        v = r.vectors[i]
        assert abs(float(v.norm()) - 1) <= 1e-12
        # (a run that exhausts the sector before the tolerance says so in its residual)
        assert float((h @ v - e * v).norm()) <= 2 * float(r.residual[i].nan_to_num()) + 1e-9 * max(1.0, abs(e))


def test_zero_and_non_finite_starts(cuda):
    from cmpy_gb300.batched import Batch

    plans = _plans("disorder")[:3]
    starts = [torch.zeros(plans[0].dim, device="cuda", dtype=torch.float64),
              torch.full((plans[1].dim,), float("nan"), device="cuda", dtype=torch.float64),
              torch.ones(plans[2].dim, device="cuda", dtype=torch.float64)]
    for cfg in (ONE[1], ONE[4], CLUSTER[2]):
        b = Batch(plans)
        b.threads, b.ctas_per_sm, b.cluster_size = cfg
        r = b.lanczos(max_steps=20, tol=0.0, check_every=0, starts=starts)
        assert r.steps.tolist()[:2] == [0, 0] and int(r.steps[2]) > 0
        assert torch.isnan(r.energy[:2]).all() and bool(torch.isfinite(r.energy[2]))
