"""Performance cases of the exact-diagonalisation framework: the calls a user's program makes,
with the sizes it makes them at, and the same results in plain 64-bit torch / numpy.

A case is a dict with a ``kind`` (which public entry point) and its sizes:

==============  ============================================================================
matvec          ``HamiltonOperator.matvec`` / ``matmat`` on GPU tensors: iterative solvers and
                time propagation written by the user
reorth          ``engine.lanczos(reorth=True)``: Heisenberg ground state, full reorthogonalisation
groundstate     ``groundstate_sector``: lowest eigenpair of one fermionic sector
lowest          ``compute_groundstate``: lowest eigenpair over all sectors of a model
gf              ``gf_continued_fraction``: zero-temperature G(z) from a ground state
sweep           ``groundstate_all_sectors``: every sector of a model in one batched launch
disorder        ``greens_functions_batched``: ground states and G(z) of many realisations
adjoint         ``greens_function_ad_batch``: G(z) of many impurity models and its gradient
thermal         ``gf_lehmann``: finite-temperature Lehmann G(z) over all sectors
tevo            ``gf_greater`` / ``gf_lesser`` / ``fourier_t2z``: real-time G(t) and G(omega)
==============  ============================================================================
"""

from __future__ import annotations

import math

import numpy as np
import torch

from cmpy_gb300 import engine as E
from cmpy_gb300.adjoint import greens_function_ad_batch
from cmpy_gb300.batched import greens_functions_batched, groundstate_all_sectors
from cmpy_gb300.exactdiag import (
    EigenState,
    compute_groundstate,
    fourier_t2z,
    gf_continued_fraction,
    gf_greater,
    gf_lehmann,
    gf_lesser,
    groundstate_sector,
)
from cmpy_gb300.models import ChainLattice, HeisenbergModel, HubbardModel, SingleImpurityAndersonModel

# Lanczos steps a ground state takes to converge, as counted by work()
GS_STEPS = 120


def listed():
    return [
        # one H*v of the smallest textbook sector (6-site open chain, 3+3 electrons, dimension
        # 400), called thousands of times by a user's own iteration: pure call latency
        dict(name="matvec_chain6", kind="matvec", model="chain", n=6, n_up=3, n_dn=3, k=1, hop=1.0, cplx=False),
        # a block of 16 vectors through an impurity model (1 + 9 star, physical fermion signs,
        # every hopping different), as block eigensolvers call it
        dict(name="matmat_siam10", kind="matvec", model="siam", n=10, n_up=5, n_dn=5, k=16, hop=0.0, cplx=False),
        # one H*v of the largest sector in use: the 14-site half-filled ring, dimension 11,778,624
        dict(name="matvec_ring14", kind="matvec", model="ring", n=14, n_up=7, n_dn=7, k=1, hop=1.0, cplx=False),
        # 20-site Heisenberg ring with random couplings, Sz = 0, 300 steps, full reorthogonalisation
        dict(name="reorth_heisenberg20", kind="reorth", n=20, s=0.0, steps=300),
        # ground state with its vector of the 14-site ring: the benchmark sector
        dict(name="groundstate_ring14", kind="groundstate", model="ring", n=14, n_up=7, n_dn=7, hop=1.0),
        # the drop-in ground-state search of the 6-site chain over all its 49 sectors
        dict(name="lowest_chain6", kind="lowest", n=6, hop=1.0),
        # local G(i w_n) of the 12-site ring, as a DMFT loop asks for it: particle and hole
        # continued fractions with 200 levels on 2048 Matsubara frequencies
        dict(name="gf_ring12", kind="gf", n=12, hop=1.0, levels=200, n_mats=2048, beta=50.0),
        # all 121 sectors of the 10-site ring at once
        dict(name="sweep_ring10", kind="sweep", n=10, hop=1.0),
        # 512 disorder realisations of the 8-site chain, sectors of uneven size, G(z) each
        dict(name="disorder_chain8", kind="disorder", n=8, count=512, levels=2000, n_real=1024, eta=0.05,
             n_mats=256, beta=10.0),
        # bath fit of 64 impurity models (1 + 9): G on the Matsubara axis and the gradient of a
        # least-squares loss; 150 levels converge the continued fractions at beta = 10
        dict(name="adjoint_siam64", kind="adjoint", bath=9, n_up=5, n_dn=5, count=64, gs_steps=250, levels=150,
             n_mats=1024, beta=10.0, signs=False),
        # thermal Lehmann G of the 6-site chain at 512 frequencies, all sectors
        dict(name="thermal_chain6", kind="thermal", n=6, hop=1.0, n_real=512, eta=0.05, beta=50.0),
        # real-time G of the 8-site chain at the default 1000 times and 2000 levels, and its
        # transform to real frequencies
        dict(name="tevo_chain8", kind="tevo", n=8, hop=1.0, num=1000, t_max=50.0, levels=2000, n_real=1000),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _near_half(rng, n):
    return min(n - 1, max(1, n // 2 + rng.choice((-1, 0, 0, 1))))


def _closed_ring(rng, n):
    """(model, n_up, n_dn) with one non-degenerate ground state: an open chain at any filling, a
    ring of even length with odd electron numbers."""
    n_up, n_dn = _near_half(rng, n), _near_half(rng, n)
    ring = n % 2 == 0 and n_up % 2 == 1 and n_dn % 2 == 1
    return ("ring" if ring else "chain"), n_up, n_dn


def draw(rng):
    kind = rng.choice(("matvec", "matvec", "reorth", "groundstate", "lowest", "gf", "sweep", "disorder", "adjoint",
                       "thermal", "tevo"))
    hop = rng.choice((1.0, 1.0, 0.5, 0.7))
    if kind == "matvec":
        model = rng.choice(("chain", "ring", "siam", "heisenberg"))
        cplx = rng.random() < 0.15
        if model == "heisenberg":
            n = rng.randint(8, 22)
            return dict(kind=kind, model=model, n=n, n_up=n // 2, n_dn=0, k=_log_int(rng, 1, 7), hop=0.0, cplx=cplx)
        n = rng.randint(5, 13)
        n_up, n_dn = _near_half(rng, n), _near_half(rng, n)
        k = _log_int(rng, 1, max(1, min(24, 11_000_000 // (math.comb(n, n_up) * math.comb(n, n_dn)))))
        return dict(kind=kind, model=model, n=n, n_up=n_up, n_dn=n_dn, k=k, hop=0.0 if model == "siam" else hop,
                    cplx=cplx)
    if kind == "reorth":
        n = rng.randint(10, 20)
        return dict(kind=kind, n=n, s=0.5 if n % 2 else float(rng.randint(0, 1)), steps=_log_int(rng, 60, 300))
    if kind == "groundstate":
        n = rng.randint(6, 13)
        model, n_up, n_dn = _closed_ring(rng, n)
        return dict(kind=kind, model=model, n=n, n_up=n_up, n_dn=n_dn, hop=hop)
    if kind == "lowest":
        return dict(kind=kind, n=rng.choice((4, 6)), hop=hop * rng.choice((1.0, 1.25)))
    if kind == "gf":
        return dict(kind=kind, n=rng.randint(6, 12), hop=hop, levels=_log_int(rng, 100, 200),
                    n_mats=_log_int(rng, 50, 2048), beta=rng.choice((10.0, 20.0, 50.0)))
    if kind == "sweep":
        return dict(kind=kind, n=rng.randint(4, 10), hop=rng.choice((1.0, 0.5, 0.25)))
    if kind == "disorder":
        return dict(kind=kind, n=rng.randint(6, 8), count=_log_int(rng, 16, 512), levels=_log_int(rng, 200, 2000),
                    n_real=_log_int(rng, 64, 1024), eta=0.1, n_mats=_log_int(rng, 32, 256), beta=10.0)
    if kind == "adjoint":
        bath = rng.randint(3, 9)
        return dict(kind=kind, bath=bath, n_up=_near_half(rng, bath + 1), n_dn=_near_half(rng, bath + 1),
                    count=_log_int(rng, 1, 64), gs_steps=200, levels=_log_int(rng, 100, 150),
                    n_mats=_log_int(rng, 100, 1024), beta=rng.choice((5.0, 10.0)), signs=rng.random() < 0.5)
    if kind == "thermal":
        return dict(kind=kind, n=rng.randint(3, 6), hop=hop, n_real=_log_int(rng, 64, 1024),
                    eta=rng.choice((0.05, 0.1)), beta=rng.choice((5.0, 20.0, 50.0)))
    return dict(kind=kind, n=rng.randint(5, 8), hop=hop, num=_log_int(rng, 200, 2000), t_max=rng.choice((20.0, 50.0)),
                levels=_log_int(rng, 300, 2000), n_real=_log_int(rng, 200, 1000))


# ---- inputs ----------------------------------------------------------------------------------


def _rng(seed):
    return np.random.default_rng(1000003 + seed)


def _u(seed):
    """Interaction of a parameter scan: a multiple of 1/8 from 2 to 8, seed by seed another one."""
    return 2.0 + (19 * seed + 5) % 49 / 8.0


def _bonds(model, n):
    if model == "siam":
        return [(0, j) for j in range(1, n)]
    b = [(i, i + 1) for i in range(n - 1)]
    return sorted(b + [(0, n - 1)]) if model == "ring" else b


def _parameters(case, seed):
    """(eps, u, hops, sign width) of a fermionic case, as its model describes itself."""
    kind, n = case["kind"], case.get("n")
    if case.get("model") == "siam":
        r = _rng(seed)
        eb, v, u = r.uniform(-2, 2, n - 1), r.uniform(0.1, 0.6, n - 1), _u(seed)
        return np.append(-u / 2, eb), np.append(u, np.zeros(n - 1)), list(v), n
    u, model = _u(seed), case.get("model", "ring" if kind in ("sweep", "gf") and n % 2 == 0 else "chain")
    return np.full(n, -u / 2), np.full(n, u), [case["hop"]] * len(_bonds(model, n)), n


def _lattice(case):
    return case.get("model", "ring" if case["kind"] in ("sweep", "gf") and case["n"] % 2 == 0 else "chain")


def _model(case, seed):
    if case.get("model") == "siam":
        eps, u, v, _ = _parameters(case, seed)
        return SingleImpurityAndersonModel(u=u[0], eps_imp=0.0, eps_bath=eps[1:], v=np.array(v), physical_signs=True)
    u = _u(seed)
    return HubbardModel(ChainLattice(case["n"], _lattice(case) == "ring"), inter=u, mu=u / 2, hop=case["hop"])


def _couplings(n, seed):
    r = _rng(seed)
    J = np.zeros((n, n))
    for i in range(n):
        k = (i + 1) % n
        J[i, k] = J[k, i] = 1.0 + 0.1 * r.standard_normal()
    return J


def _half(case):
    n = case["n"]
    return (n + 1) // 2, n // 2


def _frequencies(case):
    real = np.linspace(-10.0, 10.0, case["n_real"]) + 1j * case["eta"] if case.get("n_real") else np.zeros(0)
    mats = 1j * (2 * np.arange(case.get("n_mats", 0)) + 1) * np.pi / case["beta"]
    return np.concatenate([real, mats])


def _disorder_inputs(case, seed):
    r = _rng(seed)
    eps = r.uniform(-1, 1, (case["count"], case["n"]))
    lo, hi = (2, 5) if case["n"] == 8 else (2, case["n"] - 2)
    return eps, [(int(a), int(b)) for a, b in r.integers(lo, hi + 1, size=(case["count"], 2))]


def _adjoint_inputs(case, seed):
    """(thetas[count, P], target G[n_mats], z, bonds, sign width): theta = [eps, U, V] of a star."""
    r = _rng(seed)
    nb, B = case["bath"], case["count"]
    z = 1j * (2 * np.arange(case["n_mats"]) + 1) * np.pi / case["beta"]
    ek = r.uniform(-2, 2, 30)
    target = 1.0 / (z - np.sum(0.3**2 / (z[:, None] - ek[None, :]), axis=1))
    th = np.zeros((B, 2 * (nb + 1) + nb))
    th[:, 0] = -2.0
    th[:, 1:nb + 1] = r.uniform(-2, 2, (B, nb))
    th[:, nb + 1] = 4.0
    th[:, 2 * (nb + 1):] = r.uniform(0.1, 0.6, (B, nb))
    return th, target, z, _bonds("siam", nb + 1), nb + 1 if case["signs"] else 0


def _start(D, seed):
    return torch.rand(D, dtype=torch.float64, generator=torch.Generator(device="cpu").manual_seed(seed))


def _vectors(case, seed):
    D = _dim(case)
    g = torch.Generator(device="cuda" if torch.cuda.is_available() else "cpu").manual_seed(seed)
    shape = (D,) if case["k"] == 1 else (D, case["k"])
    x = torch.randn(shape, dtype=torch.float64, device=g.device, generator=g)
    if case["cplx"]:
        x = torch.complex(x, torch.randn(shape, dtype=torch.float64, device=g.device, generator=g))
    return x


def prepare(case, seed):
    kind = case["kind"]
    st = dict(kind=kind, case=case)
    if kind == "matvec":
        if case["model"] == "heisenberg":
            m = HeisenbergModel(ChainLattice(case["n"], True), j=_couplings(case["n"], seed))
            st["op"] = m.hamilton_operator(s=case["n_up"] - case["n"] / 2)
        else:
            m = _model(case, seed)
            st["op"] = m.hamilton_operator(case["n_up"], case["n_dn"])
        st["x"] = _vectors(case, seed)
    elif kind == "reorth":
        J = _couplings(case["n"], seed)
        st["plan"] = HeisenbergModel(ChainLattice(case["n"], True), j=J, jz=J).plan(case["s"])
        st["v0"] = _start(st["plan"].dim, seed).cuda()
    elif kind in ("groundstate", "lowest", "sweep", "thermal"):
        st["model"] = _model(case, seed)
        if kind == "groundstate":
            st["model"].plan(case["n_up"], case["n_dn"])
        if kind == "thermal":
            st["z"] = _frequencies(case)
    elif kind in ("gf", "tevo"):
        st["model"], (nu, nd) = _model(case, seed), _half(case)
        st["e0"], st["psi"] = groundstate_sector(st["model"], nu, nd)
        if kind == "gf":
            st["z"] = _frequencies(case)
        else:
            st["gs"] = EigenState(st["e0"], st["psi"], nu, nd)
            st["omegas"] = np.linspace(-8.0, 8.0, case["n_real"])
    elif kind == "disorder":
        eps, st["sectors"] = _disorder_inputs(case, seed)
        lat = ChainLattice(case["n"], False)
        st["models"] = [HubbardModel(lat, inter=4.0, eps=e, mu=2.0, hop=1.0) for e in eps]
        st["z"] = _frequencies(case)
    else:
        th, target, z, st["bonds"], st["width"] = _adjoint_inputs(case, seed)
        st["theta"] = torch.as_tensor(th).cuda().requires_grad_(True)
        st["target"] = torch.as_tensor(target).cuda()
        st["z"] = torch.as_tensor(z).cuda()
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "matvec":
        return st["op"].matvec(st["x"]) if case["k"] == 1 else st["op"].matmat(st["x"])
    if kind == "reorth":
        r = E.lanczos(st["plan"], max_steps=case["steps"], reorth=True, want_vector=True, v0=st["v0"])
        return {"energy": r.energy, "vector": r.vector}
    if kind == "groundstate":
        e, v = groundstate_sector(st["model"], case["n_up"], case["n_dn"])
        return {"energy": e, "vector": v}
    if kind == "lowest":
        gs = compute_groundstate(st["model"])
        return {"energy": gs.energy, "n_up": gs.n_up, "n_dn": gs.n_dn, "state": gs.state}
    if kind == "gf":
        nu, nd = _half(case)
        g = gf_continued_fraction(st["model"], st["z"], nu, nd, st["e0"], st["psi"], pos=0, n_lev=case["levels"])
        return g
    if kind == "sweep":
        _, res, _ = groundstate_all_sectors(st["model"])
        return {"energies": res.energy}
    if kind == "disorder":
        e, g = greens_functions_batched(st["models"], st["sectors"], st["z"], gf_levels=case["levels"])
        return {"energies": e, "g": g}
    if kind == "adjoint":
        g = greens_function_ad_batch(st["theta"], case["bath"] + 1, st["bonds"], (case["n_up"], case["n_dn"]), st["z"],
                                     sign_width=st["width"], gs_steps=case["gs_steps"], gf_levels=case["levels"])
        loss = torch.sum(torch.abs(g - st["target"]) ** 2)
        (grad,) = torch.autograd.grad(loss, st["theta"])
        return {"g": g.detach(), "grad": grad}
    if kind == "thermal":
        d = gf_lehmann(st["model"], st["z"], case["beta"])
        return {"g": d.gf, "occ": d.occ, "occ_double": d.occ_double, "energy": d.gs_energy}
    t, gg = gf_greater(st["model"], st["gs"], 0.0, case["t_max"], case["num"], n_lev=case["levels"])
    _, gl = gf_lesser(st["model"], st["gs"], 0.0, case["t_max"], case["num"], n_lev=case["levels"])
    _, gw = fourier_t2z(t, gg - gl, st["omegas"])
    return {"greater": gg, "lesser": gl, "gw": gw}


# ---- work ------------------------------------------------------------------------------------


def _sector(n, k):
    return math.comb(n, k) if 0 <= k <= n else 0


def _dim(case):
    n = case["n"]
    return _sector(n, case["n_up"]) * (1 if case.get("model") == "heisenberg" else _sector(n, case["n_dn"]))


def _hops(n, k, nb):
    """Single-particle hops (non-zeros) of one spin species with nb bonds."""
    return nb * 2 * math.comb(n - 2, k - 1) if 0 < k < n else 0


def _nnz(n, nu, nd, nb):
    """Non-zeros of a fermionic sector, the diagonal counted once."""
    D = _sector(n, nu) * _sector(n, nd)
    return D + _hops(n, nu, nb) * _sector(n, nd) + _hops(n, nd, nb) * _sector(n, nu)


def _lanczos_work(D, nnz, steps):
    """Per step: read the vector, read the previous one, write the next; 2 flops a non-zero and
    the recurrence's dot, two updates and norm."""
    steps = min(steps, D)
    return np.array([24.0 * D * steps, (2.0 * nnz + 8.0 * D) * steps])


def _gf_work(n, nu, nd, nb, levels):
    w = np.zeros(2)
    for d in (1, -1):
        D = _sector(n, nu + d) * _sector(n, nd)
        if D:
            w += _lanczos_work(D, _nnz(n, nu + d, nd, nb), levels)
    return w


def work(case):
    kind, n = case["kind"], case.get("n")
    nb = n if n and kind in ("sweep", "gf") and n % 2 == 0 else (n or 1) - 1
    if kind == "matvec":
        D, k = _dim(case), case["k"] * (2 if case["cplx"] else 1)
        if case["model"] == "heisenberg":
            nnz = D + _hops(n, case["n_up"], n)
        else:
            nnz = _nnz(n, case["n_up"], case["n_dn"], len(_bonds(case["model"], n)))
        w = np.array([16.0 * D * k, 2.0 * nnz * k])
    elif kind == "reorth":
        D = math.comb(n, int(n / 2 + case["s"]))
        m = min(case["steps"], D)
        w = _lanczos_work(D, D + _hops(n, int(n / 2 + case["s"]), n), m)
        # two Gram-Schmidt passes over the basis so far, each vector used in a dot and an update
        w += np.array([2 * 8.0, 2 * 4.0]) * D * m * (m + 1) / 2
    elif kind == "groundstate":
        D = _dim(case)
        nnz = _nnz(n, case["n_up"], case["n_dn"], len(_bonds(case["model"], n)))
        w = _lanczos_work(D, nnz, GS_STEPS) + np.array([8.0 * D * GS_STEPS, 2.0 * D * GS_STEPS])
    elif kind in ("lowest", "sweep"):
        w = np.zeros(2)
        for a in range(n + 1):
            for b in range(n + 1):
                w += _lanczos_work(_sector(n, a) * _sector(n, b), _nnz(n, a, b, nb), GS_STEPS)
    elif kind == "gf":
        nu, nd = _half(case)
        nz = case["n_mats"]
        w = _gf_work(n, nu, nd, nb, case["levels"]) + np.array([32.0 * nz, 2 * 12.0 * case["levels"] * nz])
    elif kind == "tevo":
        nu, nd = _half(case)
        w = _gf_work(n, nu, nd, nb, case["levels"])
        w += np.array([48.0 * case["num"] + 32.0 * case["n_real"],
                       2 * 20.0 * case["levels"] * case["num"] + 30.0 * case["num"] * case["n_real"]])
    elif kind == "disorder":
        _, sectors = _disorder_inputs(case, 0)
        nz = case["n_real"] + case["n_mats"]
        w = np.array([16.0 * nz * case["count"], 2 * 12.0 * case["levels"] * nz * case["count"]])
        for a, b in sectors:
            w += _lanczos_work(_sector(n, a) * _sector(n, b), _nnz(n, a, b, nb), GS_STEPS)
            w += _gf_work(n, a, b, nb, case["levels"])
    elif kind == "adjoint":
        n, nb, B = case["bath"] + 1, case["bath"], case["count"]
        nu, nd = case["n_up"], case["n_dn"]
        steps = _lanczos_work(_sector(n, nu) * _sector(n, nd), _nnz(n, nu, nd, nb), GS_STEPS)
        # forward, and in the reverse sweep each step recomputed and transposed
        w = 3.0 * B * (steps + _gf_work(n, nu, nd, nb, case["levels"]))
        w += B * case["n_mats"] * np.array([32.0, 6 * 12.0 * case["levels"]])
    else:  # thermal: eigenpairs of every sector (4/3 n^3 + 2 n^3 flops), overlaps and pole sums
        w = np.zeros(2)
        for a in range(n + 1):
            for b in range(n + 1):
                D, Dp = _sector(n, a) * _sector(n, b), _sector(n, a + 1) * _sector(n, b)
                w += np.array([8.0 * D * D, 10.0 / 3.0 * D**3])
                w += np.array([8.0 * D * Dp, 2.0 * D * D * Dp + 8.0 * D * Dp * case["n_real"]])
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ---- the same results in plain torch / numpy ----------------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _states(n, k):
    s = np.arange(1 << n, dtype=np.int64)
    pop = np.zeros_like(s)
    for i in range(n):
        pop += (s >> i) & 1
    return s[pop == k]


def _hop_lists(n, k, bonds, hops, width):
    """(idx[S, m], coef[S, m]) of one spin species, rows padded with (own index, 0)."""
    st = _states(n, k)
    S, rows = len(st), np.arange(len(st))
    idx, coef = [], []
    for (i, j), t in zip(bonds, hops):
        sel = ((st >> i) ^ (st >> j)) & 1 == 1
        tgt = np.where(sel, np.searchsorted(st, st ^ (1 << i) ^ (1 << j)), rows)
        par = np.zeros(S, dtype=np.int64)
        for b in range(i + 1, j):
            if b < width:
                par ^= (st >> b) & 1
        idx.append(tgt)
        coef.append(np.where(sel, np.where(par == 1, -t, t), 0.0))
    if not idx:
        return st, np.zeros((S, 0), np.int64), np.zeros((S, 0))
    order = np.argsort(np.stack(coef, 1) == 0, axis=1, kind="stable")
    I, C = np.take_along_axis(np.stack(idx, 1), order, 1), np.take_along_axis(np.stack(coef, 1), order, 1)
    m = int((C != 0).sum(1).max()) if S else 0
    return st, I[:, :m], C[:, :m]


class _Fermions:
    """H of one fermionic sector on [n_up states, n_dn states, ...] arrays."""

    def __init__(self, n, nu, nd, eps, u, bonds, hops, width):
        self.dev = _dev()
        self.up, iu, cu = _hop_lists(n, nu, bonds, hops, width)
        self.dn, id_, cd = _hop_lists(n, nd, bonds, hops, width)
        bit = lambda s, i: ((s >> i) & 1).astype(np.float64)
        e = lambda s: sum((bit(s, i) * eps[i] for i in range(n)), np.zeros(len(s)))
        diag = e(self.up)[:, None] + e(self.dn)[None, :]
        for i in range(n):
            if u[i]:
                diag += u[i] * bit(self.up, i)[:, None] * bit(self.dn, i)[None, :]
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(self.dev)
        self.diag, self.iu, self.cu, self.id, self.cd = t(diag), t(iu), t(cu), t(id_), t(cd)
        self.shape = (len(self.up), len(self.dn))
        self.dim = self.shape[0] * self.shape[1]
        self._mats = None

    def single(self):
        """Dense single-spin hopping matrices."""
        if self._mats is None:
            out = []
            for idx, c in ((self.iu, self.cu), (self.id, self.cd)):
                a = torch.zeros((idx.shape[0], idx.shape[0]), dtype=torch.float64, device=self.dev)
                if idx.shape[1]:
                    a.scatter_add_(1, idx, c)
                out.append(a)
            self._mats = out
        return self._mats

    def apply(self, x):
        """H x for one vector."""
        X = x.reshape(self.shape)
        y = self.diag * X
        if max(self.shape) <= 1000:
            a, b = self.single()
            y += a @ X
            y += X @ b.t()
        else:
            for k in range(self.iu.shape[1]):
                y += self.cu[:, k, None] * X[self.iu[:, k]]
            for k in range(self.id.shape[1]):
                y += self.cd[None, :, k] * X[:, self.id[:, k]]
        return y.reshape(-1)

    def dense(self):
        a, b = self.single()
        h = torch.kron(a, torch.eye(self.shape[1], dtype=torch.float64, device=self.dev))
        h += torch.kron(torch.eye(self.shape[0], dtype=torch.float64, device=self.dev), b)
        return h + torch.diag(self.diag.reshape(-1))

    def terms(self, X):
        """The products of H X on [n_up, n_dn, k] arrays, as (coefficient, array) pairs."""
        yield self.diag[..., None], X
        for k in range(self.iu.shape[1]):
            yield self.cu[:, k, None, None], X[self.iu[:, k]]
        for k in range(self.id.shape[1]):
            yield self.cd[None, :, k, None], X[:, self.id[:, k]]


class _Spins:
    """H of the Heisenberg ring: pairs (i, i+1), each in both directions."""

    def __init__(self, n, n_up, J):
        self.dev = _dev()
        bonds = sorted({(min(i, (i + 1) % n), max(i, (i + 1) % n)) for i in range(n)})
        st, idx, coef = _hop_lists(n, n_up, bonds, [0.25 * J[i, j] for i, j in bonds], 0)
        diag = np.zeros(len(st))
        for i, j in bonds:
            diag += 0.5 * J[i, j] * np.where(((st >> i) ^ (st >> j)) & 1 == 0, 1.0, -1.0)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(self.dev)
        self.diag, self.idx, self.coef = t(diag), t(idx), t(coef)
        self.dim = len(st)
        self.shape = (self.dim, 1)

    def apply(self, x):
        y = self.diag * x
        for k in range(self.idx.shape[1]):
            y += self.coef[:, k] * x[self.idx[:, k]]
        return y

    def terms(self, X):
        yield self.diag[:, None, None], X
        for k in range(self.idx.shape[1]):
            yield self.coef[:, k, None, None], X[self.idx[:, k]]


def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _two_prod(a, b):
    def split(v):
        c = 134217729.0 * v
        h = c - (c - v)
        return h, v - h

    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _apply_exact(h, x):
    """H x with every product and sum carried in two doubles."""
    X = x.to(h.dev).reshape(h.shape + (-1,))
    hi = torch.zeros_like(X)
    lo = torch.zeros_like(X)
    for c, g in h.terms(X):
        p, e = _two_prod(c, g)
        hi, r = _two_sum(hi, p)
        lo += r + e
    return (hi + lo).reshape(x.shape)


def _krylov(h, v, steps, keep):
    """Lanczos (alpha, beta, basis or None) from v; with `keep` every vector is orthogonalised
    twice against the whole basis."""
    q = v.to(h.dev) / torch.linalg.norm(v)
    steps = min(steps, h.dim)
    Q = torch.zeros((steps, h.dim), dtype=torch.float64, device=h.dev) if keep else None
    al, be, prev, b = [], [], None, None
    for k in range(steps):
        if keep:
            Q[k] = q
        w = h.apply(q)
        a = torch.dot(q, w)
        al.append(a)
        w -= a * q
        if prev is not None:
            w -= b * prev
        if keep:
            for _ in range(2):
                w -= Q[:k + 1].t() @ (Q[:k + 1] @ w)
        b = torch.linalg.norm(w)
        if k + 1 < steps:
            be.append(b)
            # the host looks at the norm now and then: an exhausted Krylov space ends the run
            if (k % 10 == 9 or h.dim <= 2 * steps) and not float(b) > 1e-10:
                be.pop()
                break
        prev, q = q, w / b
    f = lambda t: torch.stack(t).cpu().numpy() if t else np.zeros(0)
    return f(al), f(be), Q


def _tri(al, be):
    m = len(al)
    return np.diag(al) + np.diag(be[:m - 1], 1) + np.diag(be[:m - 1], -1)


def _lowest(h, v=None, steps=160, vector=False):
    if h.dim <= 400 and hasattr(h, "dense"):
        w, V = torch.linalg.eigh(h.dense())
        return float(w[0]), V[:, 0].contiguous()
    v = _start(h.dim, 0) if v is None else v
    keep = h.dim <= 1_000_000
    al, be, Q = _krylov(h, v, steps if keep else 200, keep)
    w, c = np.linalg.eigh(_tri(al, be))
    if not vector:
        return float(w[0]), None
    psi = torch.as_tensor(c[:, 0]).to(h.dev) @ Q[:len(al)]
    return float(w[0]), psi / torch.linalg.norm(psi)


def _neighbour(n, nu, nd, par, bonds, psi, up, delta):
    """(H, vector) of c^dag_0 (delta = 1) or c_0 (delta = -1) on psi: site 0 passes no other."""
    eps, u, hops, width = par
    if not 0 <= nu + delta <= n:
        return None, None
    h = _Fermions(n, nu + delta, nd, eps, u, bonds, hops, width)
    occ = h.up & 1 == (1 if delta > 0 else 0)
    src = np.searchsorted(up, h.up[occ] ^ 1)
    phi = torch.zeros(h.shape, dtype=torch.float64, device=h.dev)
    phi[torch.as_tensor(np.nonzero(occ)[0]).to(h.dev)] = psi.reshape(len(up), -1)[torch.as_tensor(src).to(h.dev)]
    return h, phi.reshape(-1)


def _spectral(n, nu, nd, par, bonds, e0, psi, up, levels):
    """[(sign, |phi|^2, alpha, beta)] of the particle and the hole Krylov spaces."""
    out = []
    for delta in (1, -1):
        h, phi = _neighbour(n, nu, nd, par, bonds, psi, up, delta)
        if h is None or h.dim == 0:
            continue
        n2 = float(torch.dot(phi, phi))
        if n2 > 0:
            al, be, _ = _krylov(h, phi, levels, True)
            out.append((delta, n2, al, be))
    return out


def _green(parts, e0, z):
    g = np.zeros(len(z), dtype=np.complex128)
    for sign, n2, al, be in parts:
        zz = sign * z + e0
        t = zz - al[-1]
        for k in range(len(al) - 2, -1, -1):
            t = zz - al[k] - be[k] ** 2 / t
        g += sign * n2 / t
    return g


def _exact_thermal(case, seed):
    n, beta, z = case["n"], case["beta"], _frequencies(case)
    eps, u, hops, width = _parameters(case, seed)
    bonds = _bonds(_lattice(case), n)
    sectors, eig = {}, {}
    for a in range(n + 1):
        for b in range(n + 1):
            h = sectors[a, b] = _Fermions(n, a, b, eps, u, bonds, hops, width)
            w, v = np.linalg.eigh(h.dense().cpu().numpy())
            eig[a, b] = (w, v)
    # the sums run over the sectors that have an upper sector
    pairs = [k for k in sectors if k[0] < n]
    e0 = min(eig[k][0][0] for k in pairs)
    weight = lambda k: np.exp(-beta * (eig[k][0] - e0))
    part = sum(weight(k).sum() for k in pairs)
    g, occ, dbl = np.zeros(len(z), dtype=np.complex128), 0.0, 0.0
    for a, b in pairs:
        h, hp = sectors[a, b], sectors[a + 1, b]
        (w, v), (wp, vp) = eig[a, b], eig[a + 1, b]
        V = v.reshape(h.shape + (-1,))
        C = np.zeros(hp.shape + (h.dim,))
        sel = hp.up & 1 == 1
        C[sel] = V[np.searchsorted(h.up, hp.up[sel] ^ 1)]
        ov = (vp.T @ C.reshape(hp.dim, -1)) ** 2 * (weight((a, b))[None, :] + weight((a + 1, b))[:, None])
        pole = (wp[:, None] - w[None, :]).reshape(-1)
        ov = ov.reshape(-1)
        pt, ot = torch.as_tensor(pole).to(_dev()), torch.as_tensor(ov).to(_dev()).to(torch.complex128)
        for i in range(0, len(z), 64):
            zt = torch.as_tensor(z[i:i + 64]).to(_dev())
            g[i:i + 64] += torch.sum(ot[None, :] / (zt[:, None] - pt[None, :]), dim=1).cpu().numpy()
        up, dn = h.up & 1, h.dn & 1
        n0 = (V[up == 1] ** 2).sum(axis=(0, 1))
        occ += np.dot(weight((a, b)), n0)
        dbl += np.dot(weight((a, b)), ((V ** 2) * (up[:, None] & dn[None, :])[..., None]).sum(axis=(0, 1)))
    return {"g": g / part, "occ": occ / part, "occ_double": dbl / part, "energy": e0}


def _exact_tevo(case, seed):
    n, (nu, nd) = case["n"], _half(case)
    par, bonds = _parameters(case, seed), _bonds(_lattice(case), n)
    h = _Fermions(n, nu, nd, par[0], par[1], bonds, par[2], par[3])
    e0, psi = _lowest(h, vector=True)
    t = np.linspace(0.0, case["t_max"], case["num"])
    out = {}
    for sign, n2, al, be in _spectral(n, nu, nd, par, bonds, e0, psi, h.up, min(case["levels"], 600)):
        w, c = np.linalg.eigh(_tri(al, be))
        out[sign] = -1j * sign * n2 * (np.exp(-1j * sign * np.outer(t, w - e0)) @ c[0] ** 2)
    zero = np.zeros(len(t), dtype=np.complex128)
    gg, gl = out.get(1, zero), out.get(-1, zero)
    # Laplace transform of the piecewise-linear interpolant on the uniform time grid
    g, dt = gg - gl, t[1] - t[0]
    omega = np.linspace(-8.0, 8.0, case["n_real"])
    uu = 1j * (omega + 1j * -np.log(1e-2) / t[-1])
    x = uu * dt
    small = np.abs(x) < 0.5
    xs = np.where(small, x, 0.1)
    xl = np.where(small, 1.0, x)
    p1 = np.where(small, sum(xs**k / math.factorial(k + 1) for k in range(24)), np.expm1(xl) / xl)
    p2 = np.where(small, sum(xs**k / math.factorial(k + 2) for k in range(24)), (np.expm1(xl) - xl) / xl**2)
    F = np.exp(np.outer(uu, t[:-1]))
    return {"greater": gg, "lesser": gl, "gw": dt * (p2 * (F @ g[:-1]) + (p1 - p2) * (F @ g[1:]))}


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "matvec":
        if case["model"] == "heisenberg":
            h = _Spins(n, case["n_up"], _couplings(n, seed))
        else:
            eps, u, hops, width = _parameters(case, seed)
            h = _Fermions(n, case["n_up"], case["n_dn"], eps, u, _bonds(case["model"], n), hops, width)
        x = _vectors(case, seed)
        if case["cplx"]:
            return torch.complex(_apply_exact(h, x.real.contiguous()), _apply_exact(h, x.imag.contiguous()))
        return _apply_exact(h, x)
    if kind == "reorth":
        h = _Spins(n, int(n / 2 + case["s"]), _couplings(n, seed))
        al, be, _ = _krylov(h, _start(h.dim, seed), case["steps"], True)
        return {"energy": float(np.linalg.eigvalsh(_tri(al, be))[0]), "vector": None}
    if kind == "thermal":
        return _exact_thermal(case, seed)
    if kind == "tevo":
        return _exact_tevo(case, seed)
    if kind == "adjoint":
        th, _, z, bonds, width = _adjoint_inputs(case, seed)
        n, nu, nd = case["bath"] + 1, case["n_up"], case["n_dn"]
        if case["count"] * math.comb(n, nu) * math.comb(n, nd) > 4_100_000 or _dev().type == "cpu":
            return None
        g = []
        for row in th:
            par = (row[:n], row[n:2 * n], list(row[2 * n:]), width)
            h = _Fermions(n, nu, nd, par[0], par[1], bonds, par[2], width)
            e0, psi = _lowest(h, steps=200, vector=True)
            g.append(_green(_spectral(n, nu, nd, par, bonds, e0, psi, h.up, case["levels"]), e0, z))
        return {"g": np.stack(g), "grad": None}
    if kind == "disorder":
        if _dev().type == "cpu":
            return None
        eps, sectors = _disorder_inputs(case, seed)
        bonds = _bonds("chain", n)
        e = [_lowest(_Fermions(n, a, b, v - 2.0, np.full(n, 4.0), bonds, [1.0] * len(bonds), n), steps=140)[0]
             for v, (a, b) in zip(eps, sectors)]
        return {"energies": np.array(e), "g": None}
    eps, u, hops, width = _parameters(case, seed)
    bonds = _bonds(_lattice(case), n)
    sector = lambda a, b: _Fermions(n, a, b, eps, u, bonds, hops, width)
    if kind == "sweep":
        # spin up and spin down enter alike: (a, b) and (b, a) have the same energies
        e = {(a, b): _lowest(sector(a, b))[0] for a in range(n + 1) for b in range(a, n + 1)}
        return {"energies": np.array([e[min(a, b), max(a, b)] for a in range(n + 1) for b in range(n + 1)])}
    if kind == "lowest":
        e = {(a, b): float(torch.linalg.eigvalsh(sector(a, b).dense())[0])
             for a in range(n + 1) for b in range(n + 1)}
        k = min(e, key=e.get)
        return {"energy": e[k], "n_up": k[0], "n_dn": k[1], "state": None}
    if kind == "groundstate":
        if _dev().type == "cpu" and _dim(case) > 1_000_000:
            return None
        return {"energy": _lowest(sector(case["n_up"], case["n_dn"]))[0], "vector": None}
    # gf
    nu, nd = _half(case)
    h = sector(nu, nd)
    e0, psi = _lowest(h, vector=True)
    parts = _spectral(n, nu, nd, (eps, u, hops, width), bonds, e0, psi, h.up, case["levels"])
    return _green(parts, e0, _frequencies(case))
