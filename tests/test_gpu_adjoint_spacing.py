"""The spacing of the batched adjoint's checkpoints: the caller's is taken as given, the choice that is left to the
library changes no bit of G or its gradient, and calls without a gradient keep no tape of the neighbours."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(requires_grad=True):
    sites, B = 6, 5
    g = torch.Generator("cuda").manual_seed(3)
    bonds = [(0, i) for i in range(1, sites)]
    th = torch.rand((B, 2 * sites + len(bonds)), dtype=torch.float64, device="cuda", generator=g) + 0.2
    z = 1j * torch.linspace(0.1, 6.0, 33, dtype=torch.float64, device="cuda").to(torch.complex128)
    return th.requires_grad_(requires_grad), sites, bonds, z


def _call(th, sites, bonds, z, **kw):
    from cmpy_gb300 import adjoint as A

    return A.greens_function_ad_batch(th, sites, bonds, (3, 3), z, gs_steps=60, gf_levels=40, **kw)


def _spacings(monkeypatch):
    from cmpy_gb300 import adjoint as A

    seen, plain = [], A.batch_tape_forward
    monkeypatch.setattr(A, "batch_tape_forward", lambda *a, **k: (seen.append(plain(*a, **k)), seen[-1])[1])
    return seen


@pytest.mark.parametrize("ckpt", [1, 5, 16, 256])
def test_as_given_and_same_bits(cuda, monkeypatch, ckpt):
    from cmpy_gb300 import adjoint as A

    th, *rest = _problem()
    seen = _spacings(monkeypatch)
    got = []
    for kw in ({}, dict(ckpt=ckpt)):
        g = _call(th, *rest, **kw)
        (grad,) = torch.autograd.grad(torch.sum(torch.abs(g - 0.1) ** 2), th)
        got.append((g.detach(), grad))
    assert [t.c for t in seen] == 3 * [A.TAPE_ALL] + 3 * [ckpt]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


def test_without_gradient(cuda, monkeypatch):
    from cmpy_gb300 import adjoint as A

    seen = _spacings(monkeypatch)
    ref = _call(*_problem())
    with torch.no_grad():
        a = _call(*_problem())
    b = _call(*_problem(False))
    assert torch.equal(ref.detach(), a) and torch.equal(a, b) and not b.requires_grad
    assert [t.c for t in seen] == 3 * [A.TAPE_ALL] + 2 * [A.TAPE_ALL, 16, 16]


def test_refused_and_default(cuda):
    import inspect

    from cmpy_gb300 import adjoint as A

    assert inspect.signature(A.greens_function_ad_batch).parameters["ckpt"].default == 16
    th, *rest = _problem()
    for ckpt in (0, -1, 257, 1 << 30):
        with pytest.raises(Exception):
            _call(th, *rest, ckpt=ckpt)
