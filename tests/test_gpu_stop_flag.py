"""A convergence test on the side stream stops a run while its step kernels are in flight: the runs of every
matvec kernel stop at the same step, time after time, with the residual that the test promised."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 2, 3, 4, 5, 6, 7, "f64", "reorth"])
def test_stopped_runs(cuda, variant):
    from cmpy_gb300 import engine as E

    n = 10
    bonds = [(i, i + 1, 1.0) for i in range(n - 1)] + [(0, n - 1, 1.0)]
    p = E.Plan.fermion(n, [-2.0] * n, [4.0] * n, bonds, 5, 5)
    kw = dict(arithmetic="fixed") if isinstance(variant, int) else dict(arithmetic="f64", reorth=variant == "reorth")
    if isinstance(variant, int):
        p.set_matvec_variant(variant)
    tol = 1e-7
    runs = [E.lanczos(p, max_steps=150, tol=tol, check_every=1 + i % 3 * 2, want_vector=True, **kw) for i in range(9)]
    for r, again in zip(runs[:3], runs[3:6]):
        assert r.converged == 1 and r.steps < 150
        assert (r.steps, r.energy) == (again.steps, again.energy)
        # |beta_m c_m| is the residual norm up to the rounding of H v and of the Ritz vector (||H|| < 64)
        limit = tol * max(1.0, abs(r.energy))
        assert r.residual <= limit
        assert float(torch.linalg.vector_norm(p.matvec(r.vector) - r.energy * r.vector)) <= limit + 1e-11
