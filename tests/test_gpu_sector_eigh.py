"""Eigenpairs of many sectors in the same launches (packed matrices of very different orders) against
one sector at a time: the three forms of the reduction (orders up to 128, up to 640, above), one state,
degenerate spectra, several chunks. Residuals and orthogonality 1e-11, eigenvalues 1e-12 of the
spectral radius (the bounds of the one-matrix solver)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plans(fillings, n, u=4.0, extra=()):
    from cmpy_gb300 import engine as E

    hop = [(i, i + 1, 1.0) for i in range(n - 1)]
    return [E.Plan.fermion(n, [-u / 2] * n, [u] * n, hop, a, b) for a, b in fillings] + list(extra)


@pytest.mark.parametrize("case", ["all6", "one", "forms", "spin"])
@pytest.mark.parametrize("chunk", [1 << 30, 200_000])
def test_packed(cuda, case, chunk):
    from cmpy_gb300 import engine as E

    if case == "all6":
        plans = _plans([(a, b) for a in range(7) for b in range(7)], 6)
    elif case == "one":
        plans = _plans([(0, 0)], 3)
    elif case == "forms":  # 784, 700 | 441, 245 | 128..1
        plans = _plans([(2, 2), (0, 3), (1, 6), (2, 1), (4, 0)], 8) + _plans([(3, 1), (3, 2)], 7) + _plans([(1, 1)], 2)
    else:
        plans = [E.Plan.spin(n, [(i, i + 1, 1.0, 1.0) for i in range(n - 1)], n // 2) for n in (4, 9, 7)]
    seen = set()
    for part in E.sector_eigh(plans, chunk):
        for i, w, v in part:
            seen.add(i)
            h = plans[i].dense()
            wr, vr = E.dense_eigh(h)
            sc = max(1.0, float(wr.abs().max()))
            assert v.stride() == vr.stride() and v.shape == vr.shape
            assert float((w - wr).abs().max()) <= 1e-12 * sc
            assert float((h @ v - v * w).abs().max()) <= 1e-11 * sc
            # (close eigenvalues that are no cluster: the solver's own 1.01e-11 at 784 states)
            eye = torch.eye(len(w), dtype=v.dtype, device=v.device)
            assert float((v.t() @ v - eye).abs().max()) <= max(1e-11, 2 * float((vr.t() @ vr - eye).abs().max()))
    assert seen == set(range(len(plans)))


def test_refusals(cuda):
    import ctypes as C

    from cmpy_gb300 import _native as N
    from cmpy_gb300 import engine as E

    plans = _plans([(1, 1), (2, 2)], 4)  # ascending: refused
    w = torch.empty(100, dtype=torch.float64, device="cuda")
    z = torch.empty(5000, dtype=torch.float64, device="cuda")
    h = (C.c_void_p * 2)(*[p.handle for p in plans])
    assert N.lib().ed_sector_eigh(h, 2, N.ptr(w), N.ptr(z), None) != N.ED_OK
    assert N.lib().ed_sector_eigh(h, 0, N.ptr(w), N.ptr(z), None) != N.ED_OK
    assert list(E.sector_eigh([])) == []
