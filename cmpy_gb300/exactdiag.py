"""Exact-diagonalisation drivers — drop-in for ``cmpy.exactdiag`` (cmpy/exactdiag.py).

* ``compute_groundstate`` (exactdiag.py:24-43): every (n_up, n_dn) sector, dense eigh for
  dim <= thresh, otherwise the device Lanczos (replacing ARPACK ``eigsh``).
* ``solve_sector`` / ``gf_lehmann`` / ``GreensFunctionMeasurement`` (exactdiag.py:46-245):
  thermal Lehmann sum with dense sector eigenproblems, the c^dag application, overlaps and
  the pole sum all on the GPU.
* ``gf_continued_fraction``: zero-temperature G(z) from Lanczos coefficients of c^dag|gs>
  and c|gs> (no reference counterpart; the reference's dense Lanczos helpers are
  exactdiag.py:324-375, mirrored below on the device).
"""

from __future__ import annotations

import logging
from typing import NamedTuple, Optional

import numpy as np
import torch

from . import engine as E
from .basis import DN, UP, Sector
from .models import AbstractManyBodyModel

logger = logging.getLogger("cmpy_gb300")

__all__ = [
    "EigenState",
    "compute_groundstate",
    "solve_sector",
    "occupation_up",
    "occupation_dn",
    "occupation",
    "double_occupation",
    "accumulate_gf",
    "GreensFunctionMeasurement",
    "gf_lehmann",
    "gf_lehmann_zero_temperature",
    "gf_continued_fraction",
    "greens_lehmann",
    "gf_lehmann_offdiag",
    "gf_greater",
    "gf_lesser",
    "gf_tevo",
    "fourier_t2z",
    "iter_lanczos_coeffs",
    "lanczos_coeffs",
    "lanczos_matrix",
    "lanczos_ground_state",
]


class EigenState(NamedTuple):
    """Ground-state record (cmpy/matrix.py:42-47)."""

    energy: float = np.inf
    state: np.ndarray = None
    n_up: int = None
    n_dn: int = None


def _dense_eigh(plan: E.Plan):
    """Every eigenpair of a sector's dense Hamiltonian (solve_sector, exactdiag.py:46-57),
    with the library's own FP64 eigensolver."""
    return E.dense_eigh(plan.dense())


def _sector_plan(model, n_up, n_dn) -> E.Plan:
    return model.plan(n_up, n_dn)


def groundstate_sector(model, n_up: int, n_dn: int, thresh: int = 50, max_steps: int = 400,
                       tol: float = 1e-12, check_every: int = 10):
    """(energy, device ground-state vector) of one sector."""
    plan = _sector_plan(model, n_up, n_dn)
    D = plan.dim
    if D <= thresh:
        w, v = _dense_eigh(plan)
        i = int(torch.argmin(w).item())
        return float(w[i].item()), v[:, i].contiguous()
    res = E.lanczos(plan, max_steps=min(max_steps, D), want_vector=True, tol=tol, check_every=check_every)
    return res.energy, res.vector


def _resident_energies(model, fillings, max_steps: int, tol: float, check_every: int = 10):
    """{filling: (energy, None)} of the sectors whose Lanczos runs fit a cluster's shared memory, all in
    one launch; the same start vectors as groundstate_sector's. The cluster of a sector is as large as
    keeps every sector's running at once (a single run: 400 states 5.6 us a step on 2 CTAs, 5.8 on 8;
    4900 states 12.6, 8.2, 7.7 on 2, 4, 8), or the smallest that still holds the largest sector's vectors:
    the 80 sectors of the 9-site chain (15,876 states at most, one CTA to an SM) on clusters of 2, whose
    vectors are in global memory, 6.95 ms, of 4, not all at once, 5.72, of 8 10.64."""
    from .batched import Batch

    n = model.num_sites
    small = [f for f in fillings if E.sector_size(n, f[0]) * E.sector_size(n, f[1]) <= 1 << 15]
    pairs = [(f, p) for f, p in zip(small, model.plans(small)) if p.resident]
    if len(pairs) < 2:
        return {}
    batch = Batch([p for _, p in pairs])
    dmax = max(batch.dims)
    sms = torch.cuda.get_device_properties(E.device()).multi_processor_count
    # (two CTAs to an SM while the vectors of the largest sector, 10 bytes a state on 8 CTAs, leave room for two)
    batch.threads, batch.ctas_per_sm = 512, 2 if dmax <= 8000 else 1
    fits = [c for c in (8, 4, 2) if batch.resident(512, batch.ctas_per_sm, c)] or [8]
    batch.cluster_size = next((c for c in fits if len(pairs) * c <= sms * batch.ctas_per_sm), fits[-1])
    x = E.random_start(dmax)
    res = batch.lanczos(min(max_steps, dmax), tol, check_every, starts=[x[:d] for d in batch.dims])
    return {f: (energy, None) for (f, _), energy in zip(pairs, res.energy.tolist())}


def compute_groundstate(model, thresh: int = 50, max_steps: int = 400, tol: float = 1e-12) -> EigenState:
    """Lowest eigenstate over all sectors (cmpy/exactdiag.py:24-43)."""
    gs = EigenState()
    best_vec = None
    fillings = list(model.basis.iter_fillings())
    n = model.num_sites
    dense = [f for f in fillings if E.sector_size(n, f[0]) * E.sector_size(n, f[1]) <= thresh]
    solved = {}
    # the dense sectors in the same launches (28 sectors of the 6-site chain: 6.2 -> 0.8 ms of kernels)
    for part in E.sector_eigh(model.plans(dense)):
        energies = torch.stack([w[0] for _, w, _ in part]).tolist()
        for (i, _, v), energy in zip(part, energies):
            solved[dense[i]] = energy, v[:, 0].contiguous()
    solved.update(_resident_energies(model, [f for f in fillings if f not in solved], max_steps, tol))
    for n_up, n_dn in fillings:
        if (n_up, n_dn) in solved:
            energy, vec = solved[n_up, n_dn]
        else:
            energy, vec = groundstate_sector(model, n_up, n_dn, thresh, max_steps, tol)
        logger.debug("Sector (%d, %d): E0 = %.12f", n_up, n_dn, energy)
        if energy < gs.energy:
            gs = EigenState(energy, None, n_up, n_dn)
            best_vec = vec
    if gs.n_up is not None and best_vec is None:
        energy, best_vec = groundstate_sector(model, gs.n_up, gs.n_dn, thresh, max_steps, tol)
        gs = gs._replace(energy=energy)
    if best_vec is not None:
        gs = gs._replace(state=best_vec.cpu().numpy())
    return gs


def _solve_sector_dev(model, sector: Sector, cache: dict = None):
    key = (sector.n_up, sector.n_dn)
    if cache is not None and key in cache:
        w, v = cache[key]
        return E._as_dev_f64(w), E._strided_dev_f64(v)
    w, v = _dense_eigh(_sector_plan(model, sector.n_up, sector.n_dn))
    if cache is not None:
        cache[key] = [w, v]
    return w, v


def _solve_sectors_dev(model, keys, cache: dict):
    """The eigenpairs of every sector of ``keys`` that the cache lacks, many sectors to a launch."""
    missing = [k for k in dict.fromkeys(keys) if k not in cache]
    for part in E.sector_eigh(model.plans(missing)):
        for i, w, v in part:
            cache[missing[i]] = [w, v]


def _lehmann_sectors(model, sigma, cache: dict):
    """The pairs (sector, sector with one particle more) of a Lehmann sum, their eigenpairs in the cache."""
    pairs = []
    for n_up, n_dn in model.basis.iter_fillings():
        upper = model.basis.upper_sector(n_up, n_dn, sigma)
        if upper is not None:
            pairs.append((model.get_sector(n_up, n_dn), upper))
    _solve_sectors_dev(model, [(s.n_up, s.n_dn) for pair in pairs for s in pair], cache)
    return pairs


def solve_sector(model: AbstractManyBodyModel, sector: Sector, cache: dict = None):
    """Dense eigenpairs of one sector (cmpy/exactdiag.py:46-57), computed on the GPU."""
    w, v = _solve_sector_dev(model, sector, cache)
    return w.cpu().numpy(), v.cpu().numpy()


# -- thermal observables (cmpy/exactdiag.py:60-107), on the device --------------------------


def _state_masks(up_states, dn_states):
    dev = E.device()
    up = torch.as_tensor(np.asarray(up_states, dtype=np.int64)).to(dev)
    dn = torch.as_tensor(np.asarray(dn_states, dtype=np.int64)).to(dev)
    return up, dn


def _weights(evals, beta, emin):
    return torch.exp(-beta * (E._as_dev_f64(evals) - emin))


def occupation_up(up_states, dn_states, evals, evecs, beta, emin, pos):
    up, dn = _state_masks(up_states, dn_states)
    V = E._as_dev_f64(evecs).reshape(len(up), len(dn), -1)
    sel = ((up >> pos) & 1).bool()
    overlap = (V[sel] ** 2).sum(dim=(0, 1))
    return float((_weights(evals, beta, emin) * overlap).sum().item())


def occupation_dn(up_states, dn_states, evals, evecs, beta, emin, pos):
    up, dn = _state_masks(up_states, dn_states)
    V = E._as_dev_f64(evecs).reshape(len(up), len(dn), -1)
    sel = ((dn >> pos) & 1).bool()
    overlap = (V[:, sel] ** 2).sum(dim=(0, 1))
    return float((_weights(evals, beta, emin) * overlap).sum().item())


def occupation(up_states, dn_states, evals, evecs, beta, emin=0.0, pos=0, sigma=UP):
    if sigma == UP:
        return occupation_up(up_states, dn_states, evals, evecs, beta, emin, pos)
    return occupation_dn(up_states, dn_states, evals, evecs, beta, emin, pos)


def double_occupation(up_states, dn_states, evals, evecs, beta, emin, pos):
    up, dn = _state_masks(up_states, dn_states)
    V = E._as_dev_f64(evecs).reshape(len(up), len(dn), -1)
    both = (((up[:, None] & dn[None, :]) >> pos) & 1).bool()
    overlap = (V[both] ** 2).sum(dim=0)
    return float((_weights(evals, beta, emin) * overlap).sum().item())


def accumulate_gf(gf, z, cdag, evals, evecs, evals_p1, evecs_p1, beta, emin=0.0):
    """gf += Lehmann poles of one sector pair (cmpy/exactdiag.py:110-134). `cdag` is a
    CreationOperator (its device map is used); `gf` is a complex128 torch CUDA tensor."""
    V = E._strided_dev_f64(evecs)  # (the solver's eigenvectors are rows in memory, as the map takes them)
    Vp = E._strided_dev_f64(evecs_p1)
    CV = cdag._apply_dev(V)
    ov = (Vp.t() @ CV) ** 2
    return E.lehmann_accumulate(evals, evals_p1, ov, float(beta), float(emin), z, gf)


class GreensFunctionMeasurement:
    """Running thermal Lehmann accumulation (cmpy/exactdiag.py:137-212)."""

    def __init__(self, z, beta, pos=0, sigma=UP, dtype=None, measure_occ=True):
        self.z = z
        self.beta = beta
        self.pos = pos
        self.sigma = sigma
        self._measure_occ = measure_occ
        self._zt = E._as_dev_c128(z)
        self._part = 0.0
        self._gs_energy = np.inf
        self._gf = torch.zeros_like(self._zt)
        self._occ = 0.0
        self._occ_double = 0.0

    @property
    def part(self):
        return self._part * np.exp(-self.beta * self._gs_energy)

    @property
    def gf(self):
        g = (self._gf / self._part).cpu().numpy()
        return g.reshape(np.shape(self.z)) if np.ndim(self.z) else g

    @property
    def occ(self):
        return self._occ / self._part

    @property
    def occ_double(self):
        return self._occ_double / self._part

    @property
    def gs_energy(self):
        return self._gs_energy

    def accumulate(self, sector, sector_p1, evals, evecs, evals_p1, evecs_p1, cdag):
        evals_t = E._as_dev_f64(evals)
        up, dn = sector.up_states, sector.dn_states
        min_energy, part, occ, double = E.thermal_sums(evals_t, evecs, up, dn, self.pos, self.sigma != UP, self.beta,
                                                       self._gs_energy, self._measure_occ)
        factor = 1.0
        if min_energy < self._gs_energy:
            factor = float(np.exp(-self.beta * (self._gs_energy - min_energy)))
            self._gs_energy = min_energy
        e0 = self._gs_energy
        self._part = self._part * factor + part
        if factor != 1.0:
            self._gf *= factor
        accumulate_gf(self._gf, self._zt, cdag, evals_t, evecs, evals_p1, evecs_p1, self.beta, e0)
        if self._measure_occ:
            self._occ = self._occ * factor + occ
            self._occ_double = self._occ_double * factor + double


def gf_lehmann(model, z, beta, pos=0, sigma=UP, eig_cache=None, occ=True, jw_sign: bool = False):
    """Thermal Lehmann Green's function over all sectors (cmpy/exactdiag.py:215-245)."""
    from .operators import CreationOperator

    basis = model.basis
    data = GreensFunctionMeasurement(z, beta, pos, sigma, measure_occ=occ)
    eig_cache = eig_cache if eig_cache is not None else dict()
    for sector, sector_p1 in _lehmann_sectors(model, sigma, eig_cache):
        w, v = _solve_sector_dev(model, sector, eig_cache)
        wp, vp = _solve_sector_dev(model, sector_p1, eig_cache)
        cdag = CreationOperator(sector, sector_p1, pos=pos, sigma=sigma, jw_sign=jw_sign)
        data.accumulate(sector, sector_p1, w, v, wp, vp, cdag)
    return data


def _lehmann_pair(model, z, beta, i, j, sigma, eig_cache, jw_sign):
    """Running Lehmann accumulation over all sectors with an upper sector (the structure of
    lehmann_full.py:48-97 and exactdiag.py:215-245) with the overlap <n|c_i|m><m|c^dag_j|n>;
    returns (gf, part), part being the partition function relative to the running E0."""
    from .operators import CreationOperator

    basis = model.basis
    eig_cache = eig_cache if eig_cache is not None else dict()
    zt = E._as_dev_c128(z)
    gf = torch.zeros_like(zt)
    part = 0.0
    e0 = np.inf
    for sector, sector_p1 in _lehmann_sectors(model, sigma, eig_cache):
        w, v = _solve_sector_dev(model, sector, eig_cache)
        wp, vp = _solve_sector_dev(model, sector_p1, eig_cache)
        w_t = E._as_dev_f64(w)
        min_energy = float(w_t.min().item())
        factor = 1.0
        if min_energy < e0:
            factor = float(np.exp(-beta * (e0 - min_energy)))
            e0 = min_energy
        part = part * factor + float(torch.exp(-beta * (w_t - e0)).sum().item())
        if factor != 1.0:
            gf *= factor
        V = E._strided_dev_f64(v)
        Vp = E._strided_dev_f64(vp)
        a_i = Vp.t() @ CreationOperator(sector, sector_p1, pos=i, sigma=sigma, jw_sign=jw_sign)._apply_dev(V)
        if j == i:
            ov = a_i**2
        else:
            a_j = Vp.t() @ CreationOperator(sector, sector_p1, pos=j, sigma=sigma, jw_sign=jw_sign)._apply_dev(V)
            ov = a_i * a_j  # <n|c_i|m><m|c^dag_j|n> (real eigenvectors)
        E.lehmann_accumulate(w_t, wp, ov, float(beta), e0, zt, gf)
    return gf, part


def greens_lehmann(model, z, beta, i, j, sigma=UP, occ=True, eig_cache=None, jw_sign: bool = False):
    """Lehmann sum of the reference's G_ij draft (lehmann_full.py:48-97), completed: the
    overlap is <n|c_i|m><m|c^dag_j|n>, and like the draft the sum is returned without dividing
    by the partition function. The draft itself computes neither G_ij nor G_ii: its sector loop
    variable shadows `i` (the operator acts on site = sector index) and the c^dag_j factor is
    commented out (lehmann_full.py:19-25, 63-90)."""
    gf, _ = _lehmann_pair(model, z, beta, i, j, sigma, eig_cache, jw_sign)
    return gf.cpu().numpy()


def gf_lehmann_offdiag(model, z, beta, i, j, sigma=UP, eig_cache=None, jw_sign: bool = False):
    """Thermal G_ij(z) = Z^-1 sum_{n,m} <n|c_i|m><m|c^dag_j|n> (e^{-beta E_n} + e^{-beta E_m}) /
    (z - E_m + E_n) over all sectors; i = j gives gf_lehmann(pos=i)."""
    gf, part = _lehmann_pair(model, z, beta, i, j, sigma, eig_cache, jw_sign)
    return (gf / part).cpu().numpy()


def _neighbour(model, n_up, n_dn, sigma, delta):
    nu, nd = (n_up + delta, n_dn) if sigma == UP else (n_up, n_dn + delta)
    if not (0 <= nu <= model.num_sites and 0 <= nd <= model.num_sites):
        return None
    return nu, nd


def gf_lehmann_zero_temperature(model, z, gs_energy: float, gs_state, n_up: int, n_dn: int, pos=0, sigma=UP,
                                jw_sign: bool = False) -> np.ndarray:
    """T=0 Lehmann G(z) of a non-degenerate ground state from the dense eigenpairs of the two
    neighbouring sectors: sum_m |<m|c^dag|0>|^2/(z-E_m+E0) + sum_n |<n|c|0>|^2/(z+E_n-E0)."""
    plan = _sector_plan(model, n_up, n_dn)
    psi = E._as_dev_f64(gs_state).reshape(-1)
    zt = E._as_dev_c128(z)
    g = torch.zeros_like(zt)
    e0 = torch.tensor([gs_energy], dtype=torch.float64, device=E.device())
    parts = []
    for delta, create in ((1, True), (-1, False)):
        nb = _neighbour(model, n_up, n_dn, sigma, delta)
        if nb is not None:
            tplan = _sector_plan(model, *nb)
            parts.append((create, tplan, plan.apply_fermion(tplan, pos, sigma, create, psi, jw_sign=jw_sign)))
    # both neighbouring sectors in one call of the eigensolver
    eig = E.dense_eigh_batch([tp.dense() for _, tp, _ in parts])
    for (create, _, phi), (w, v) in zip(parts, eig):
        amp = (v.t() @ phi) ** 2  # |<m|phi>|^2
        if create:  # poles at E_m - E0, weights amp (Lehmann with unit ground-state weight)
            E.lehmann_accumulate(e0, w, amp.reshape(-1, 1), float("inf"), 0.0, zt, g)
        else:  # poles at E0 - E_n:  1/(z - (E0 - E_n))
            E.lehmann_accumulate(w, e0, amp.reshape(1, -1), float("inf"), 0.0, zt, g)
    # unit weights (beta=inf) add w_n + w'_m = 2 per pole; undo that factor
    return (g / 2).cpu().numpy()


def gf_continued_fraction(model, z, n_up: int, n_dn: int, gs_energy: float, gs_state, pos=0, sigma=UP,
                          n_lev: int = 200, jw_sign: bool = False, return_coeffs: bool = False):
    """T=0 G(z) = <0|c (z-H+E0)^-1 c^dag|0> + <0|c^dag (z+H-E0)^-1 c|0> from the Lanczos
    continued fractions of c^dag|0> and c|0>, evaluated on the device for every z."""
    plan = _sector_plan(model, n_up, n_dn)
    psi = E._as_dev_f64(gs_state).reshape(-1)
    zt = E._as_dev_c128(z)
    g = torch.zeros_like(zt)
    coeffs = {}
    parts = []
    for delta, create, sign in ((1, True, 1), (-1, False, -1)):
        nb = _neighbour(model, n_up, n_dn, sigma, delta)
        if nb is None:
            continue
        tplan = _sector_plan(model, *nb)
        parts.append((create, sign, tplan, plan.apply_fermion(tplan, pos, sigma, create, psi, jw_sign=jw_sign)))
    if parts:
        # the particle and the hole run in one call: their steps interleave on the GPU
        K = min(n_lev, max(tp.dim for _, _, tp, _ in parts))
        runs = E.lanczos_coeffs_multi([(tp, phi) for _, _, tp, phi in parts], max_steps=K)
        for (create, sign, _, _), (a, b, nrm) in zip(parts, runs):
            coeffs["particle" if create else "hole"] = (a, b, nrm)
            if a.numel() == 0:
                continue
            E.continued_fraction(a, b, nrm * nrm, zt, e0=gs_energy, sign=sign, out=g)
    out = g.cpu().numpy()
    return (out, coeffs) if return_coeffs else out


# -- real-time Green's functions (cmpy/exactdiag.py:248-316) -------------------------------


def _tevo_levels(plan, times: np.ndarray) -> int:
    """Lanczos levels that <phi|exp(-iHt)|phi> can depend on to FP64 rounding. T_m and T_M, M > m, give the
    same moments up to degree 2 m - 1, and exp(-iHt) is a polynomial of degree N = z + 14 z^(1/3) + 40
    to 1e-17 on an interval that holds H's spectrum, of half-width z / |t| (the coefficients of its
    Chebyshev expansion are Bessel functions J_k(z)). 8-site chain, |t| <= 50: 643 levels, not 2000 (the run
    11.5 -> 3.7 ms)."""
    lo, hi = plan.spectrum_bounds()
    z = 0.5 * (hi - lo) * float(np.max(np.abs(times), initial=0.0))
    return int(np.ceil(0.5 * (z + 14.0 * np.cbrt(z) + 41.0))) if z < 8192.0 else 4096


def _tevo_part(model, gs, times: np.ndarray, pos: int, sigma: int, delta: int, n_lev: Optional[int],
               jw_sign: bool) -> Optional[torch.Tensor]:
    """-i e^{iE0 t}<gs|c e^{-iHt} c^dag|gs> (delta=+1) or +i e^{-iE0 t}<gs|c^dag e^{iHt} c|gs>
    (delta=-1) on the device. The reference propagates with scipy expm_multiply; here the
    Lanczos tridiagonal T_m of the start vector gives <phi|e^{-iHt}|phi> = |phi|^2 e1^T
    e^{-iT_m t} e1, evaluated by a Chebyshev expansion in T_m (exact once m reaches the dimension,
    and converged long before that for ||H|| t << m)."""
    nb = _neighbour(model, gs.n_up, gs.n_dn, sigma, delta)
    if nb is None:
        return None
    plan = _sector_plan(model, gs.n_up, gs.n_dn)
    tplan = _sector_plan(model, *nb)
    psi = E._as_dev_f64(gs.state).reshape(-1)
    phi = plan.apply_fermion(tplan, pos, sigma, delta > 0, psi, jw_sign=jw_sign)
    steps = tplan.dim if n_lev is None else min(int(n_lev), tplan.dim)
    if steps <= 4096:
        steps = min(steps, _tevo_levels(tplan, times))
    a, b, nrm = E.lanczos_coeffs(tplan, phi, max_steps=steps)
    m = a.numel()
    if m == 0 or nrm == 0.0:
        return torch.zeros(len(times), dtype=torch.complex128, device=E.device())
    return E.tevo_krylov(a, b, nrm * nrm, float(gs.energy), 1 if delta > 0 else -1, times)


def _tevo(model, gs, start, stop, num, pos, sigma, delta, n_lev, jw_sign):
    times = np.linspace(start, stop, num)
    g = _tevo_part(model, gs, times, pos, sigma, delta, n_lev, jw_sign)
    if g is None:
        logger.warning("%s sector not found!", "Upper" if delta > 0 else "Lower")
        return times, np.zeros_like(times)
    return times, g.cpu().numpy()


def gf_greater(model, gs, start, stop, num=1000, pos=0, sigma=UP, n_lev: Optional[int] = 2000,
               jw_sign: bool = False):
    """Greater Green's function -i e^{i E0 t} <gs|c e^{-iHt} c^dag|gs> at `num` times in
    [start, stop] (cmpy/exactdiag.py:248-273). n_lev caps the Krylov dimension (None: the
    sector dimension)."""
    return _tevo(model, gs, start, stop, num, pos, sigma, +1, n_lev, jw_sign)


def gf_lesser(model, gs, start, stop, num=1000, pos=0, sigma=UP, n_lev: Optional[int] = 2000,
              jw_sign: bool = False):
    """Lesser Green's function +i e^{-i E0 t} <gs|c^dag e^{iHt} c|gs> (cmpy/exactdiag.py:276-301)."""
    return _tevo(model, gs, start, stop, num, pos, sigma, -1, n_lev, jw_sign)


def gf_tevo(model, start, stop, num=1000, pos=0, sigma=UP, n_lev: Optional[int] = 2000):
    """G(t) = G^>(t) - G^<(t) of the ground state (cmpy/exactdiag.py:304-308)."""
    gs = compute_groundstate(model)
    times, gg = gf_greater(model, gs, start, stop, num, pos, sigma, n_lev)
    _, gl = gf_lesser(model, gs, start, stop, num, pos, sigma, n_lev)
    return times, gg - gl


def fourier_t2z(times, gf_t, omegas, delta=1e-2, eta=None, method: str = "lin"):
    """G(z) = int e^{izt} G(t) dt at z = omega + i eta, eta = -ln(delta)/t_last by default
    (cmpy/exactdiag.py:311-316). The reference calls gftool.fourier.tt2z; its default rule,
    the exact integral of the piecewise-linear interpolant of G(t), is evaluated on the device
    ("trapz" selects the trapezoidal rule)."""
    times = np.asarray(times, dtype=np.float64)
    if eta is None:
        eta = -np.log(delta) / times[-1]
    z = np.asarray(omegas) + 1j * eta
    gw = E.laplace_t2z(times, gf_t, z, method=method)
    return z, gw.cpu().numpy()


# -- Lanczos helpers (cmpy/exactdiag.py:324-375) on the device ------------------------------


def _as_operator_dev(ham):
    from .operators import HamiltonOperator

    if isinstance(ham, HamiltonOperator):
        return ham._apply_dev
    H = E._as_dev_f64(ham)
    return lambda x: H @ x


def iter_lanczos_coeffs(ham, size=10, seed: Optional[int] = None):
    """Un-normalised Lanczos (a_n, b_n) with a uniform(0,1) start, no reorthogonalisation
    (cmpy/exactdiag.py:324-347), on the device."""
    apply = _as_operator_dev(ham)
    n = ham.shape[0]
    g = torch.Generator(device="cpu")
    if seed is not None:
        g.manual_seed(int(seed))
    psi = torch.rand(n, generator=g, dtype=torch.float64).to(E.device())
    hpsi = apply(psi)
    a = torch.dot(psi, hpsi) / torch.dot(psi, psi)
    yield float(a.item()), None
    psi_prev, psi = psi, hpsi - a * psi
    for _ in range(1, size):
        hpsi = apply(psi)
        pp = torch.dot(psi, psi)
        a = torch.dot(psi, hpsi) / pp
        b2 = pp / torch.dot(psi_prev, psi_prev)
        psi_new = hpsi - a * psi - b2 * psi_prev
        yield float(a.item()), float(torch.sqrt(b2).item())
        psi_prev, psi = psi, psi_new


def lanczos_coeffs(ham, size=10, seed: Optional[int] = None):
    a_coeffs, b_coeffs = [], []
    for a, b in iter_lanczos_coeffs(ham, size, seed):
        a_coeffs.append(a)
        b_coeffs.append(b)
    b_coeffs.pop(0)
    return a_coeffs, b_coeffs


def lanczos_matrix(a_coeffs, b_coeffs):
    mat = np.diag(a_coeffs)
    np.fill_diagonal(mat[1:], b_coeffs)
    np.fill_diagonal(mat[:, 1:], b_coeffs)
    return mat


def lanczos_ground_state(a_coeffs, b_coeffs, max_eig=3):
    """Lowest eigenpair of the Lanczos tridiagonal matrix, solved on the device
    (cmpy/exactdiag.py:368-375)."""
    a = np.asarray(a_coeffs, dtype=np.float64)
    b = np.concatenate([[0.0], np.asarray(b_coeffs, dtype=np.float64)])
    e, v = E.tridiag_lowest(a, b, want_vector=True)
    return e, v.cpu().numpy()
