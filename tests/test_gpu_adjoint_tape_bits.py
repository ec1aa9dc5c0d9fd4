"""The whole batched tape and the checkpointed one give the same bits: which of them a call takes depends on the
memory that is free, its results must not."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites, up, dn, B, K", [(2, 1, 0, 1, 3), (4, 2, 1, 3, 12), (6, 3, 3, 6, 40), (7, 4, 3, 9, 70)])
@pytest.mark.parametrize("c", [1, 7, 16])
def test_same_bits(cuda, monkeypatch, sites, up, dn, B, K, c):
    from cmpy_gb300 import adjoint as A

    g = torch.Generator("cuda").manual_seed(sites)
    bonds = [(0, i) for i in range(1, sites)]
    P = 2 * sites + len(bonds)
    th = torch.rand((B, P), dtype=torch.float64, device="cuda", generator=g) + 0.2
    plan = A.structure_plan(sites, bonds, sites, up, dn)
    starts = torch.rand((B, plan.dim), dtype=torch.float64, device="cuda", generator=g)
    if B > 1:
        starts[0] = 0.0  # an empty tape
        h = A.plan_from_params(th[1], sites, bonds, sites, up, dn).dense()
        starts[1] = torch.linalg.eigh(h)[1][:, :3].sum(1)  # a short one
    got = []
    for spacing in (lambda *_: A.TAPE_ALL, lambda c, *_: c):
        monkeypatch.setattr(A, "_tape_spacing", spacing)
        t = A.batch_tape_forward(plan, th, A.batch_diag(plan, th), starts, K, c)
        r = torch.Generator("cuda").manual_seed(1)
        rnd = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=r)  # noqa: E731
        bar = torch.zeros((B, P), dtype=torch.float64, device="cuda")
        sbar = A.batch_tape_reverse(t, rnd(B, t.K), rnd(B, t.K + 1), bar, ext_coef=rnd(B, t.K), ext_vec=rnd(B, plan.dim))
        got.append((bar, sbar))
    live = [b for b in range(B) if t.m[b] > 0]
    for x, y in zip(*got):
        assert torch.equal(x[live], y[live]) and bool(torch.isfinite(y[live]).all())
