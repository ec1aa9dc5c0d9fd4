"""The expansion of the real-time G leaves Krylov coefficients that are not finite to the eigenpairs: it reports so and
writes nothing."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 7, 300])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
def test_left_to_the_eigenpairs(cuda, m, bad):
    from cmpy_gb300 import _native as N
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(m)
    t = torch.linspace(0, 3, 17, dtype=torch.float64, device="cuda")

    def run(a, b):
        g = torch.full((17,), 0.5 + 2j, dtype=torch.complex128, device="cuda")
        done = C.c_int(7)
        N.check(N.lib().ed_tevo_krylov(N.ptr(a), N.ptr(b), m, 1.0, 0.0, 1, N.ptr(t), 17, 3.0,
                                       N.ptr(torch.view_as_real(g)), 0, C.byref(done), E._stream()))
        return done.value, g

    a, b = (torch.as_tensor(x).cuda() for x in (r.uniform(-1, 1, m), r.uniform(0.1, 1, m)))
    assert run(a, b)[0] == 1
    for i in {0, m // 2, m - 1}:
        wrong = a.clone()
        wrong[i] = bad
        done, g = run(wrong, b)
        assert done == 0 and bool((g == 0.5 + 2j).all())
        if i > 0:  # (beta[0] is not used)
            wrong = b.clone()
            wrong[i] = bad
            done, g = run(a, wrong)
            assert done == 0 and bool((g == 0.5 + 2j).all())
