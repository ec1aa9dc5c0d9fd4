"""The Krylov basis stays orthogonal when the second Gram-Schmidt pass runs only where the first found
something: max |Q^T Q - I| < 1e-14 (always two passes: 2.2e-15 at most), in sectors that a run exhausts, with
a start vector in a small invariant subspace and one next to it (there the second pass runs), and in
large units."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _orthogonality(p, K, v0=None):
    from cmpy_gb300 import engine as E

    ws = torch.empty((K + 8) * p.dim * 16 + (64 << 20), dtype=torch.uint8, device="cuda")
    r = E.lanczos(p, max_steps=K, reorth=True, want_vector=True, seed=3, v0=v0, workspace=ws, arithmetic="f64")
    Q = ws[: r.steps * p.dim * 8].view(torch.float64).view(r.steps, p.dim)
    eye = torch.eye(r.steps, dtype=torch.float64, device="cuda")
    return r, float((Q @ Q.t() - eye).abs().max())


def _chain(n, scale=1.0):
    return [-2.0 * scale] * n, [4.0 * scale] * n, [(i, i + 1, scale) for i in range(n - 1)]


@pytest.mark.parametrize("which", ["heisenberg", "hubbard", "siam", "units", "exhausted"])
def test_orthogonal(cuda, which):
    from cmpy_gb300 import engine as E

    if which == "heisenberg":
        p, K = E.Plan.spin(12, [(i, i + 1, 1.0, 1.0) for i in range(11)], 6), 300
    elif which == "hubbard":
        p, K = E.Plan.fermion(8, *_chain(8), 4, 4), 250
    elif which == "siam":
        p, K = E.Plan.fermion(6, [-2.0, -1, -0.5, 0, 0.5, 1], [4.0] + [0.0] * 5,
                              [(0, i, 0.3 + 0.05 * i) for i in range(1, 6)], 3, 3), 400
    elif which == "units":
        p, K = E.Plan.fermion(7, *_chain(7, 2.0**60), 4, 3), 200
    else:
        p, K = E.Plan.fermion(4, *_chain(4), 2, 2), 100
    r, err = _orthogonality(p, K)
    assert err < 1e-14
    if p.dim <= 1300:
        e = np.linalg.eigvalsh(p.dense().cpu().numpy())[0]
        assert abs(r.energy - e) < 1e-12 * max(1.0, abs(e))


@pytest.mark.parametrize("eps", [0.0, 1e-13, 1e-9, 1e-4])
def test_invariant_subspace(cuda, eps):
    from cmpy_gb300 import engine as E

    p = E.Plan.fermion(6, *_chain(6), 3, 2)
    w, v = np.linalg.eigh(p.dense().cpu().numpy())
    rng = np.random.default_rng(0)
    x = v[:, [0, 40, 90]].sum(axis=1) + eps * rng.standard_normal(p.dim)
    r, err = _orthogonality(p, 60, torch.as_tensor(x).cuda())
    assert err < 1e-14 and r.steps >= 3
    assert abs(r.energy - w[0]) < 1e-12 * abs(w[0])
