"""The division-free continued fraction against an extended-precision evaluation: tile edges, one
level, frequencies on and near the real axis and far away (the recurrence's range), zero couplings, and
the batched forms."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(a, b, n2, z, e0, sign):
    """(value, condition): backwards in extended precision; the condition sums how far a relative
    rounding of each level moves the value."""
    zz = sign * z.astype(np.clongdouble) + np.longdouble(e0)
    t = zz - np.longdouble(a[-1])
    ts = [t]
    for k in range(len(a) - 2, -1, -1):
        t = zz - np.longdouble(a[k]) - np.longdouble(b[k + 1]) ** 2 / t
        ts.append(t)
    ts = ts[::-1]
    amp, cond = np.ones(len(z)), np.zeros(len(z))
    for k, t in enumerate(ts):
        scale = np.abs(zz) + abs(a[k]) + (b[k + 1] ** 2 / np.abs(ts[k + 1]) if k + 1 < len(ts) else 0)
        cond = cond + amp * (scale / np.abs(t)).astype(float)
        if k + 1 < len(ts):
            amp = amp * (b[k + 1] ** 2 / np.abs(t) / np.abs(ts[k + 1])).astype(float)
    return (sign * n2 / ts[0]).astype(complex), cond


def _z():
    return np.concatenate([np.linspace(-12, 12, 101) + 0.05j, 1j * np.array([1e-3, 0.3, 50.0]),
                           [1e9 + 1j, -1e30 + 1e28j, 3e60j, 0.1 + 1e-6j]])


@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 700, 2000])
@pytest.mark.parametrize("sign", [1, -1])
def test_single(cuda, n, sign):
    from cmpy_gb300 import engine as E

    r = np.random.default_rng(n)
    a = r.uniform(-8, 8, n)
    b = np.concatenate([[0.0], r.uniform(0.2, 4, n)])
    if n > 300:
        b[40] = 1e-7
        b[290] = 0.0
    z = _z()
    ref, cond = _reference(a, b, 0.7, z, -1.3, sign)
    got = E.continued_fraction(a, b[:n + 1], 0.7, z, e0=-1.3, sign=sign).cpu().numpy()
    # up to eight roundings a level, each moving the value by the level's condition
    assert np.all(np.abs(got - ref) <= 8 * 2.0**-53 * (cond + 4) * np.abs(ref))
    acc = torch.as_tensor(ref).cuda()
    E.continued_fraction(a, b[:n + 1], 0.7, z, e0=-1.3, sign=sign, out=acc)
    assert torch.equal(acc, torch.as_tensor(ref).cuda() + torch.as_tensor(got).cuda())


def test_batched(cuda):
    from cmpy_gb300.batched import BatchResult, batch_cf

    r = np.random.default_rng(3)
    n, K = 7, 300
    m = np.array([1, 0, 300, 256, 2, 77, 257], dtype=np.int32)
    a, b = r.uniform(-5, 5, (n, K)), r.uniform(0.3, 2, (n, K + 1))
    e0 = r.uniform(-1, 1, n)
    t = lambda x: torch.as_tensor(x).cuda()
    for z in (_z(), _z()[:1], np.linspace(-3, 3, 129) + 0.1j):
        g = batch_cf(BatchResult(None, t(m), None, t(a), t(b), None), t(e0), -1, z).cpu().numpy()
        for p in range(n):
            if m[p] == 0:
                assert np.all(g[p] == 0)
                continue
            ref, cond = _reference(a[p, :m[p]], b[p, :m[p] + 1], b[p, 0] ** 2, z, e0[p], -1)
            assert np.all(np.abs(g[p] - ref) <= 8 * 2.0**-53 * (cond + 4) * np.abs(ref))
