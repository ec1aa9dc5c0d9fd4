"""The whole batched tape against the checkpointed one: the same Krylov vectors, and sums and gradients that
differ by the rounding of H q_k as the recurrence gives it; tapes of uneven lengths, empty ones among them."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites, up, dn, B, K", [(2, 1, 0, 1, 3), (4, 2, 1, 3, 12), (6, 3, 3, 6, 40)])
@pytest.mark.parametrize("c", [1, 5, 16])
def test_whole_tape(cuda, monkeypatch, sites, up, dn, B, K, c):
    from cmpy_gb300 import adjoint as A

    g = torch.Generator("cuda").manual_seed(sites)
    bonds = [(0, i) for i in range(1, sites)]
    P = 2 * sites + len(bonds)
    th = torch.rand((B, P), dtype=torch.float64, device="cuda", generator=g) + 0.2
    plan = A.structure_plan(sites, bonds, sites, up, dn)
    diag = A.batch_diag(plan, th)
    starts = torch.rand((B, plan.dim), dtype=torch.float64, device="cuda", generator=g)
    if B > 1:
        starts[0] = 0.0
        H = A.plan_from_params(th[1], sites, bonds, sites, up, dn).dense()
        starts[1] = torch.linalg.eigh(H)[1][:, 0]  # ends after one step
    got = []
    for spacing in (A._tape_spacing, lambda c, *_: c):
        monkeypatch.setattr(A, "_tape_spacing", spacing)
        t = A.batch_tape_forward(plan, th, diag, starts, K, c)
        assert (t.c == A.TAPE_ALL) == (not got)
        r = torch.Generator("cuda").manual_seed(1)
        rnd = lambda *s: torch.randn(s, dtype=torch.float64, device="cuda", generator=r)  # noqa: E731
        y, d = A.batch_tape_combine(t, coef=rnd(B, t.K), probe=rnd(B, plan.dim))
        bar = torch.zeros((B, P), dtype=torch.float64, device="cuda")
        sbar = A.batch_tape_reverse(t, rnd(B, t.K), rnd(B, t.K + 1), bar, ext_coef=rnd(B, t.K), ext_vec=rnd(B, plan.dim))
        got.append((t, y, torch.stack([d[b] * (torch.arange(t.K, device="cuda") < t.m[b]) for b in range(B)]), bar, sbar))
    (t0, y0, d0, b0, s0), (t1, y1, d1, b1, s1) = got
    assert t0.m == t1.m and torch.equal(t0.alpha, t1.alpha) and torch.equal(t0.beta, t1.beta)
    assert torch.equal(y0, y1) and torch.equal(d0, d1)
    # the adjoints of a run that ends at a rounding-sized beta amplify rounding: the bounds of the tape's other tests
    torch.testing.assert_close(b0, b1, rtol=1e-8, atol=1e-9 * b1.abs().max().item())
    torch.testing.assert_close(s0, s1, rtol=1e-8, atol=1e-9 * s1.abs().max().item())


def test_spacing_is_checked(cuda):
    from cmpy_gb300 import adjoint as A

    for c in (0, -3, 257, A.TAPE_ALL):
        with pytest.raises(ValueError):
            A._tape_spacing(c, 8, 4)
    assert A._tape_spacing(16, 1 << 40, 100) == 16
