"""FF_NonBonded energies and virial where an error of a constant, or a decision below
FP32 spacing, would be the same for every pair: isolated charged pairs, all at about
one distance, against the same law in 64 bits, summed exactly (math.fsum).

Allowed per evaluation: six standard deviations of the sum of N independent errors, each
of one rounding to 2^-32 kcal/mol (a work item's; at most one item a pair), 2^-44 of the
pair's terms and what a rounding of its distance (2^-47 r) makes of them.  Each case states what the planted difference amounts to, well above that."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KCAL = 4184.0 / 6.0221418e23
ECONV = (6.0221418e23 / 4184.0) * 1.60217645e-19 ** 2 / (4.0 * math.pi * 8.854187817e-12 * 1e-10)
F = np.float32


def _rest(x):
    """what two FP32 numbers leave of x"""
    h = F(x)
    return x - float(h) - float(F(x - float(h)))


def _law(r, qq, inner, cut):
    """Coulomb with the energy switch: energy and r dE/dr of pairs"""
    E = qq / r
    w = np.maximum(r - inner, 0.0)
    iw = 1.0 / (cut - inner) ** 2
    s = 1.0 - w * w * iw
    return E * s * s, -(s * s * E) + E * (-4.0 * w * iw * s) * r


def _evaluate(pos, box, q, inner, cut, far=None, lj=(0.0, 0.0)):
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    n = len(pos)
    im = SystemImage([n], box, q, np.full(n, lj[0]), np.full(n, lj[1]), np.full(n, 2e-26), np.zeros((0, 3), np.int32), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(Cutoff=cut, InnerCutoff=inner, VdwCutoff=cut, VdwInnerCutoff=inner, Vdw14Scaling=1.0, Elec14Scaling=1.0,
               Dielectric=1.0, EnergySwitch=1, ForceSwitch=0, DoVdw=1, DoElec=1)
    ctx.set_positions(pos)
    e = ctx.compute(ffi.NB)[0]
    ctx.close()
    return {k: e[k] / KCAL for k in ("vdw", "elec", "virial")}


def _allowed(n, terms, slope):
    return 6.0 * math.sqrt(n) * (0.29 * 2.0 ** -32 + 2.0 ** -44 * terms + 2.0 ** -47 * slope)


def test_virial_of_pairs_a_hair_beyond_the_inner_radius():
    """r - InnerCutoff = 2e-7 to 4.7e-7 A, below the spacing of FP32 numbers there: the
    switch's slope, 4 u / w^2 of the energy times r, counts."""
    cut, inner, N = 12.0, 10.0, 400
    rng = np.random.default_rng(3)
    site = 40.0 * np.stack(np.unravel_index(np.arange(N), (8, 8, 8)), 1)
    pos = np.repeat(site, 2, axis=0)
    pos[1::2, 0] += inner + rng.uniform(2e-7, 4.7e-7, N)
    r = pos[1::2, 0] - pos[0::2, 0]
    q = np.ones(2 * N)
    e = _evaluate(pos, np.zeros(3), q, inner, cut)
    E, vir = _law(r, ECONV, inner, cut)
    tol = _allowed(N, ECONV / inner, 4.0 * ECONV / (cut - inner) ** 2 * inner)
    assert abs(math.fsum(vir) + math.fsum(E)) > 100 * tol           # (without the slope the virial is -E)
    assert abs(e["virial"] - math.fsum(vir)) <= tol and abs(e["elec"] - math.fsum(E)) <= tol


@pytest.mark.parametrize("periodic", [0, 1])
def test_sums_of_many_pairs_at_one_distance(periodic):
    """20,000 pairs whose inner radius, or 1,600 across the faces of a box whose edge,
    is not the sum of two FP32 numbers."""
    rng = np.random.default_rng(periodic)
    if periodic:
        cand = 1203.0 + 0.01 * np.arange(400)
        L = float(max(cand, key=lambda x: abs(_rest(x))))
        inner, cut, m = 10.0, 12.0, 40
        N = m * m
        site = np.stack([np.zeros(N), *(30.0 * np.stack(np.unravel_index(np.arange(N), (m, m))))], 1)
        pos = np.repeat(site, 2, axis=0)
        pos[0::2, 0] = L - 4.0
        pos[1::2, 0] = rng.uniform(6.65, 6.75, N)
        r = pos[1::2, 0] - pos[0::2, 0] + L
        box = np.full(3, L)
    else:
        cand = 10.0 + 0.01 * np.arange(200)
        inner = float(max(cand, key=lambda x: abs(_rest(x))))
        cut, m, L = inner + 2.0, 28, 0.0
        N = 20_000
        pos = np.repeat(35.0 * np.stack(np.unravel_index(np.arange(N), (m, m, m)), 1), 2, axis=0)
        pos[1::2, 0] += inner + rng.uniform(0.15, 0.25, N)
        r = pos[1::2, 0] - pos[0::2, 0]
        box = np.zeros(3)
    e = _evaluate(pos, box, np.full(2 * N, 3.0), inner, cut)
    law = lambda r, inner: _law(r, 9.0 * ECONV, inner, cut)
    E, vir = law(r, inner)
    h = 1e-5
    slope = abs(law(r + h, inner)[1] - law(r - h, inner)[1]).mean() / (2 * h)
    tol = _allowed(N, float(np.abs(vir).max()), slope * r[0])
    planted = N * slope * abs(_rest(L if periodic else inner))   # (the switch's width is a constant of its own)
    assert planted > 2.5 * tol, (planted, tol)
    assert abs(e["virial"] - math.fsum(vir)) <= tol, (e["virial"] - math.fsum(vir), tol, planted)
    assert abs(e["elec"] - math.fsum(E)) <= tol


def test_energies_of_overlapping_atoms_are_fp64():
    """Two atoms 0.9 to 1.4 A apart: LJ energies of 1e4 to 1e6 kcal/mol to 2^-50 of
    themselves (their law in FP64: some ten roundings of 2^-53) and 2^-31 kcal/mol."""
    radius, eps = 1.6, 1.0e-11
    se2 = (eps * math.sqrt(6.0221418e23 / 4184.0)) ** 2
    for k, r in enumerate((0.9, 1.05, 1.23, 1.4)):
        for image in (0, 1):
            L = 25.3
            pos = np.array([[0.3, 0.2, 0.1], [0.3 + r, 0.2, 0.1]])
            box = np.full(3, L if image else 0.0)
            if image:
                pos[0, 0] += L
            e = _evaluate(pos, box, np.array([0.7, 0.4]), 10.0, 12.0, lj=(radius, eps))
            d = pos[1, 0] - pos[0, 0]
            d -= box[0] * np.rint(d / box[0]) if image else 0.0
            B = (2.0 * radius / abs(d)) ** 6
            for key, ref in (("vdw", se2 * (B * B - 2.0 * B)), ("elec", ECONV * 0.7 * 0.4 / abs(d)),
                             ("virial", -12.0 * se2 * (B * B - B) - ECONV * 0.7 * 0.4 / abs(d))):
                assert abs(e[key] - ref) <= 2.0 ** -49 * abs(ref) + 2.0 ** -31, (r, image, key, e[key] - ref, ref)


def test_sum_of_force_switched_pairs():
    """Coulomb with the force switch, 10,000 pairs across its shell: PD's powers of r
    (nonbonded.cpp:798-819) in extended precision.  Held as pairs of FP32 numbers, their
    constants are off by 2^-49, some 1e-14 of qq in the difference of powers, alike for every
    pair: 5e-7 kcal/mol in all."""
    cut, inner, N, m = 10.39, 9.04, 10_000, 22
    ld = np.longdouble
    if np.finfo(ld).eps > 1e-18:
        pytest.skip("no extended precision on this host")
    rng = np.random.default_rng(7)
    pos = np.repeat(30.0 * np.stack(np.unravel_index(np.arange(N), (m, m, m)), 1), 2, axis=0)
    pos[1::2, 0] += rng.uniform(inner + 0.1, cut - 0.1, N)
    r = (pos[1::2, 0] - pos[0::2, 0]).astype(ld)
    from pd_gb300 import ffi
    from pd_gb300.engine import DeviceContext
    from pd_gb300.workspace import SystemImage
    im = SystemImage([2 * N], np.zeros(3), np.full(2 * N, 3.0), np.zeros(2 * N), np.zeros(2 * N), np.full(2 * N, 2e-26),
                     np.zeros((0, 3), np.int32), pos=pos)
    ctx = DeviceContext(im)
    ctx.set_list(1.0)
    ctx.set_nb(Cutoff=cut, InnerCutoff=inner, VdwCutoff=cut, VdwInnerCutoff=inner, Vdw14Scaling=1.0, Elec14Scaling=1.0,
               Dielectric=1.0, EnergySwitch=0, ForceSwitch=1, DoVdw=1, DoElec=1)
    ctx.set_positions(pos)
    e = ctx.compute(ffi.NB)[0]["elec"] / KCAL
    ctx.close()
    C, I = ld(cut), ld(inner)
    V = lambda x: (-(C ** 6 - 3 * C ** 4 * I ** 2) / x + 6 * C * C * I * I * x - (C * C + I * I) * x ** 3 + ld(2) / 5 * x ** 5) / (
        C * C - I * I) ** 3
    qq = 9.0 * ECONV
    E = (-ld(qq) * (V(r) - V(C))).astype(np.float64)
    tol = _allowed(N, float(np.abs(E).max()), qq / inner ** 2 * cut)
    assert 5e-7 > 2.5 * tol
    assert abs(e - math.fsum(E)) <= tol, (e - math.fsum(E), tol)
