"""The fast build's merged element bodies at the edges of their range: slopes
on both sides of 2^-6 (z = 2^-12), positions on both sides of the limits and
of the aperture, momenta down to delta = -1, one and several slices, bends on
both sides of the slice angle that picks the body, against the oracle; warps
with steep lanes; times of the paths that once ran two bodies."""
import itertools

import numpy as np
import pytest

from elegant_b200 import Lattice, configs
from oracle import pyoracle
from tests.helpers import compare, gpu_run, oracle_run

pytestmark = pytest.mark.gpu
PC = configs.P_CENTRAL

# 0.8512 of the slice angle is compared with 0.010: 8 slices of 0.0117 and of 0.0118
ELEMENTS = {
    "quad": ("KQUAD", dict(L=0.3, K1=1.2, N_SLICES=3)),
    "quad_one_slice": ("KQUAD", dict(L=0.3, K1=-2.0, N_SLICES=1)),
    "sext": ("KSEXT", dict(L=0.2, K2=40.0, N_SLICES=2)),
    "oct": ("KOCT", dict(L=0.1, K3=300.0, N_SLICES=2)),
    "dipole": ("CSBEND", dict(L=1.0, ANGLE=0.0936, N_SLICES=8)),
    "dipole_unmerged": ("CSBEND", dict(L=1.0, ANGLE=0.0944, N_SLICES=8)),
    "dipole_one_slice": ("CSBEND", dict(L=0.1, ANGLE=0.008, N_SLICES=1)),
    "bend_k1": ("CSBEND", dict(L=0.8, ANGLE=0.022, K1=-0.4, N_SLICES=4)),
    "quad_radiating": ("KQUAD", dict(L=0.3, K1=1.2, N_SLICES=3, SYNCH_RAD=1)),
    "sext_radiating": ("KSEXT", dict(L=0.2, K2=40.0, N_SLICES=1, SYNCH_RAD=1)),
    "dipole_radiating": ("CSBEND", dict(L=1.0, ANGLE=0.0936, N_SLICES=8, SYNCH_RAD=1)),
    "bend_k1k2": ("CSBEND", dict(L=0.8, ANGLE=0.03, K1=0.3, K2=5.0, N_SLICES=5)),
}
APERTURES = {
    "none": None,
    "rectangle": dict(X_MAX=0.004, Y_MAX=0.003),
    "ellipse": dict(X_MAX=0.005, Y_MAX=0.004, ELLIPTICAL=1),
    "superellipse": dict(X_MAX=0.005, Y_MAX=0.004, ELLIPTICAL=1, EXPONENT=4),
}


def _beam(aperture):
    slopes = [0.0, 1e-5, -3e-3, 0.0156, -0.01563, 0.02]
    if aperture == "none":
        xs, ys, slopes = [0.0, 1e-3, -0.3, 7.99, -8.01, 9.99, 10.01], [0.0, -2e-3, 8.01], slopes + [-0.4, 0.999, 1.001]
    else:
        xs = [0.0, 1e-3, -0.0035, 0.00399, 0.004, -0.00401, 0.0049, 0.00501]
        ys = [0.0, 0.0025, -0.00299, 0.00301, -0.0039]
    rows = [(x, xp, y, yp, 0.01, d) for x, xp, y, yp, d in
            itertools.product(xs, slopes, ys, (0.0, -2e-5, 0.0155), (0.0, 3e-3, -0.4, -0.999))]
    rng = np.random.Generator(np.random.Philox(3))
    jitter = rng.normal(0.0, 1e-6, (len(rows), 6)) * [1, 1, 1, 1, 1, 0]
    rows = np.hstack([np.array(rows) + jitter, np.arange(1.0, len(rows) + 1)[:, None]])
    return rows


@pytest.mark.parametrize("aperture", sorted(APERTURES))
@pytest.mark.parametrize("name", sorted(ELEMENTS))
def test_limits_of_the_merged_bodies(tracker, name, aperture):
    kind, params = ELEMENTS[name]
    lat = Lattice()
    if APERTURES[aperture]:
        lat.add("MAXAMP", "AP", **APERTURES[aperture])
    lat.add(kind, name, **params)
    beam = _beam(aperture)
    nl, g, lp, le, _ = gpu_run(tracker, lat, beam, 1, PC, fast=True)
    with pyoracle.modes(exact_sums=True, cr_math=True):
        rows, nlo, _ = oracle_run(lat, beam, 1, PC)
    r = compare(g, rows, nl, nlo)
    assert 0 < nlo and r["same_survivors"], r
    o, gi = rows[np.argsort(rows[:, 6])], np.argsort(g[:, 6])
    lost = o[:, 7] >= 0
    assert np.array_equal(lp[gi][lost], o[lost, 7].astype(np.int64))
    assert np.array_equal(le[gi][lost], o[lost, 8].astype(np.int32))
    # each of the element's substeps rounds a few times, 2^-53 of a value of the
    # particle's own or, in the oracle's bend drift (rho0 (cos/cos - 1)), of rho0;
    # the steps after it carry the error on with a gain of at most a few
    steps = 4 * params["N_SLICES"]
    rho = params["L"] / params["ANGLE"] if kind == "CSBEND" else 1.0
    alive = ~lost
    ref, got = o[alive, :6], g[gi][alive, :6]
    # a steep slope's tangent amplifies the rounding of its momentum by 1 + slope^2
    gain = 1 + np.max(np.abs(ref[:, [1, 3]]), axis=1) ** 2
    floor = np.array([rho, 1.0, rho, 1.0, rho, 1e-300])
    bound = 20 * steps * 2.0 ** -53 * np.maximum(np.abs(ref), floor) * gain[:, None] ** 2
    # delta passes through, or changes by 1e-6 of itself in steps rounded at its own size
    bound[:, 5] = 20 * steps * 2.0 ** -53 * np.maximum(np.abs(ref[:, 5]), 1e-3) if "SYNCH_RAD" in params else 0.0
    bad = np.abs(got - ref) > bound
    assert not bad.any(), (bad.sum(axis=0), ref[bad.any(axis=1)][:3], (got - ref)[bad.any(axis=1)][:3])


@pytest.mark.parametrize("rad", [0.0, 1.0])
def test_superellipse_costs_what_an_ellipse_does(tracker, rad):
    """A beam well inside takes each element's body once, whatever the
    exponents: with a second body the superellipse took 3 (radiating: 8) times
    as long as the ellipse, with one 1.15 (1.03)."""
    ms = {}
    beam = configs.gaussian_beam(100000, seed=3)
    for exponent in (2, 4):
        lat = Lattice()
        lat.add("MAXAMP", "AP", X_MAX=0.025, Y_MAX=0.025, ELLIPTICAL=1, EXPONENT=exponent)
        lat.extend(configs.c2_lattice(cells=10, with_rf=False, with_wake=False))
        for e in lat.elements:
            if e[0] in ("KQUAD", "KSEXT", "CSBEND"):
                e[2]["SYNCH_RAD"] = rad
        ms[exponent] = min(gpu_run(tracker, lat, beam, 1, PC, fast=True)[4]["device_ms"] for _ in range(5))
    assert ms[4] < 2 * ms[2], ms


def test_entry_slope_above_the_limit_is_a_loss(tracker):
    """x' = 1.2 is a loss at the element's entry even where the kicks take
    nearly all of it away: strength and position are solved for momenta below
    1e-4 after each of the three kicks."""
    lat = Lattice()
    lat.add("KQUAD", "Q", L=0.1, K1=5604218.137052551, N_KICKS=4)
    beam = np.zeros((2, 7))
    beam[0, :2], beam[:, 6] = [-0.08107141710017259, 1.2], [1, 2]
    nl, g, lp, le, _ = gpu_run(tracker, lat, beam, 1, PC, fast=True)
    with pyoracle.modes(exact_sums=True, cr_math=True):
        rows, nlo, _ = oracle_run(lat, beam, 1, PC)
    assert compare(g, rows, nl, nlo)["same_survivors"] and nl == 1


def _line_with_steep_lanes():
    lat = configs.c5_lattice(cells=1, with_rf=False, with_wake=False)
    lat.extend(configs.c2_lattice(cells=1, with_rf=False, with_wake=False))
    return lat


@pytest.mark.parametrize("variant, rad", [(-1, 0.0), (4, 0.0), (7, 0.0), (-1, 1.0)])
def test_tracks_do_not_depend_on_steep_neighbours(tracker, variant, rad):
    """A warp with a steep lane takes the bodies that hold for steep slopes;
    its other lanes keep every bit."""
    lat = _line_with_steep_lanes()
    for e in lat.elements:
        if e[0] in ("KQUAD", "KSEXT", "CSBEND"):
            e[2]["SYNCH_RAD"], e[2]["ISR"] = rad, rad
    beam = configs.c5_beam(3000, seed=8)
    _, alone, _, _, _ = gpu_run(tracker, lat, beam, 2, PC, fast=True, variant=variant)
    mixed = beam.copy()
    mixed[::5, 1], mixed[::7, 3] = 0.018, -0.05
    _, g, _, _, _ = gpu_run(tracker, lat, mixed, 2, PC, fast=True, variant=variant)
    same = np.ones(3000, bool)
    same[::5] = same[::7] = False
    assert np.array_equal(g[np.argsort(g[:, 6])][same], alone[np.argsort(alone[:, 6])][same])


@pytest.mark.parametrize("rad", [0.0, 1.0])
def test_steep_beam_takes_one_body(tracker, rad):
    """A divergent beam (12 mrad) once ran the merged and the unmerged body of
    every element, 2.3 (radiating: 3.8) times a narrow beam's time; the wide
    bodies take 1.6 (1.3)."""
    ms = {}
    lat = configs.c2_lattice(cells=1, with_rf=False, with_wake=False)
    for e in lat.elements:
        if e[0] in ("KQUAD", "KSEXT", "CSBEND"):
            e[2]["SYNCH_RAD"], e[2]["ISR"] = rad, rad
    for slope in (0.0, 0.012):
        beam = configs.gaussian_beam(400000, seed=3)
        beam[:, 1], beam[:, 3] = beam[:, 1] * slope / 10e-6, beam[:, 3] * slope / 10e-6
        ms[slope] = min(gpu_run(tracker, lat, beam, 1, PC, fast=True)[4]["device_ms"] for _ in range(5))
    assert ms[0.012] < 2 * ms[0.0], ms


def test_kick_roundings_do_not_move_the_tune(tracker):
    """A FODO channel of 40 cells against the same integrator in extended
    precision, with the element tables' constants.  A kick's rounding, the same
    in all quadrupoles of a kind, is coherent: per particle it may be up to
    2^-54 of the slice's kick k, 3e-17 in the mean, which shifts the phase by
    beta k L/2 a quadrupole, 144 in all and 5e-15 of y.  With the roundings of
    the steps themselves 1.4e-14 is measured; three kicks of a slice rounded
    apart, up to 1.7 k large, gave 2.6e-14."""
    lat = Lattice()
    for _ in range(40):
        lat.add("KQUAD", "QF", L=0.3, K1=1.2, N_KICKS=8)
        lat.add("DRIF", "D", L=3.0)
        lat.add("KQUAD", "QD", L=0.3, K1=-1.2, N_KICKS=8)
        lat.add("DRIF", "D", L=3.0)
    beam = configs.gaussian_beam(2000, seed=20)
    _, g, _, _, _ = gpu_run(tracker, lat, beam, 1, PC, fast=True)
    g = g[np.argsort(g[:, 6])]
    x, xp, y, yp, _, dp = (beam[:, c].astype(np.longdouble) for c in range(6))
    b = 1.25992104989487316477
    drift = [0.5 / (2 - b), (1 - b) / (2 - b) / 2, (1 - b) / (2 - b) / 2, 0.5 / (2 - b)]
    kick = [1.0 / (2 - b), -b / (2 - b), 1.0 / (2 - b)]
    for kind, _, p, _ in lat.elements:
        if kind == "DRIF":
            x, y = x + p["L"] * xp, y + p["L"] * yp
            continue
        r = (1 + dp) / np.sqrt(1 + xp * xp + yp * yp)
        qx, qy = xp * r, yp * r
        for step in range(8):
            h = np.longdouble(p["L"] / 2 * drift[step % 4])
            x, y = x + xp * h, y + yp * h
            if step % 4 < 3:
                k = np.longdouble(p["K1"] * p["L"] / 2 * kick[step % 4])
                qx, qy = qx - k * x, qy + k * y
                r = 1 / np.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
                xp, yp = qx * r, qy * r
    for c, v in ((0, x), (2, y)):
        err = np.linalg.norm((g[:, c] - v).astype(float)) / np.linalg.norm(v.astype(float))
        assert err < 2e-14, (c, err)
