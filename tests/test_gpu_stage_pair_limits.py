"""The pair form where recovery leaves its common path.

The pair form decides by one test per pair which cells go through the scalar
recovery (pressure floor, |Z| cap, convergence).  The states here lie where
that decision matters and nowhere else: uniform up to a few per cent, so that
the scheme's own conditioning does not magnify rounding, and compared with the
strict form after one step by the fast arithmetic's bar of 1e-5 per component
(largest difference over largest magnitude).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_REF = np.float32(0.125)  # e_ref = a_rad of the default model
E_FLOOR = np.float32(1e-7) * E_REF
GRID = (24, 20, 18)
DIRECTION = np.array([1.0, 2.0, -2.0]) / 3.0


def _wave(grid):
    """A smooth periodic function of values within 1."""
    nx, ny, nz = grid
    z, y, x = np.meshgrid(*(2 * np.pi * np.arange(n) / n for n in (nz, ny, nx)), indexing="ij")
    return (np.sin(x) + np.sin(y + 1.0) + np.cos(z)).ravel() / 3.0


def _state(e, z, phi=0.0, pi=0.0):
    n = len(e)
    field = np.stack([np.broadcast_to(phi, n), np.broadcast_to(pi, n)], 1)
    return field.astype(np.float32), np.concatenate([np.asarray(e)[:, None], z], 1).astype(np.float32)


def _compare(bubble, grid, f0, u0, precision="single", eos="bag", eos_param=(1.0, 0.0)):
    got = {}
    for math in ("strict", "fast"):
        spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", precision=precision, math=math, eos=eos,
                                     eos_param=eos_param)
        with bubble.Simulation(spec) as sim:
            sim.load_state(f0, u0)
            sim.advance(1)
            got[math] = sim.copy_state()
    for a, s in zip(got["fast"], got["strict"]):
        a, s = np.asarray(a, np.float64), np.asarray(s, np.float64)
        assert np.isfinite(a).all() and np.isfinite(s).all()
        scale = np.max(np.abs(s), axis=0)
        scale[scale == 0] = 1.0
        err = np.max(np.abs(a - s), axis=0) / scale
        assert np.all(err <= 1e-5), err


@pytest.mark.parametrize("precision,eos,eos_param", [("single", "bag", (1.0, 0.0)), ("mixed", "bag", (1.0, 0.0)),
                                                     ("single", "gamma_law", (1.2, 0.0)),
                                                     ("single", "gamma_law", (2.0, 0.0))])
def test_momentum_beyond_the_cap_at_the_energy_floor(bubble, gpu, precision, eos, eos_param):
    """At E = e_floor the pressure floor is comparable to E, so |Z| = 1.2 E ..
    1.85 E gives |v| below the gamma = 3 threshold if it is not capped."""
    w = _wave(GRID)
    e = E_FLOOR * (1.1 + 0.05 * w)
    r = np.random.default_rng(1).choice([1.01, 1.2, 1.5, 1.85, 2.0], size=len(e))
    f0, u0 = _state(e, DIRECTION * (r * e)[:, None])
    _compare(bubble, GRID, f0, u0, precision, eos, eos_param)


@pytest.mark.parametrize("gamma,e0", [(1.2, 0.05), (2.0, 0.12), (1.02, 0.12)])
def test_gamma_law_energy_below_its_offset(bubble, gpu, gamma, e0):
    """For E below e0 c2 / (1 + c2) the quadratic of the closed form has only
    roots that are rounding errors; the pressure is the floor.  Read through
    the friction of a uniform lattice, d pi / dt = -eta W(v) pi with v = Z /
    (E + p), where nothing else acts: the flux of such a state is of the order
    of e0, and its rounding would cover Z.  |v| <= 0.9, so dW / dv <= 11 and
    the bar of 1e-5 is a hundred roundings of v."""
    grid, pi = (8, 8, 8), 1e-6
    n = grid[0] * grid[1] * grid[2]
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", eos="gamma_law", eos_param=(gamma, e0))
    got = {}
    for math in ("strict", "fast"):
        spec.math = math
        got[math] = []
        with bubble.Simulation(spec) as sim:
            for e in np.geomspace(1e-6, 1e-3, 41):
                for r in (0.01, 0.3, 0.6, 0.75, 0.9):
                    e32 = np.full(n, e, np.float32)
                    sim.load_state(*_state(e32, np.outer(r * e32, DIRECTION), pi=pi))
                    sim.advance(1)
                    got[math].append(sim.copy_state()[0][:, 1].astype(np.float64) / pi)
    err = np.max(np.abs(np.array(got["fast"]) - np.array(got["strict"])), axis=1)
    assert np.all(err <= 1e-5), (np.flatnonzero(err > 1e-5), err.max())


THERMAL = [(0.0125, 0.05), (0.999 * 0.125 / 6.0, 0.999 * 0.125 / np.sqrt(2.0))]


def _thermal_energy(gamma, T, phi):
    return 0.125 * T**4 - 0.5 * gamma * (T * phi) ** 2


def _pi_after_a_step(bubble, states, eos_param, pi):
    """pi of uniform lattices (e, |Z|, phi) after one step, strict and fast."""
    grid, n = (8, 8, 8), 512
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", eos="thermal", eos_param=eos_param)
    got = {}
    for math in ("strict", "fast"):
        spec.math = math
        got[math] = []
        with bubble.Simulation(spec) as sim:
            for e, z, phi in states:
                sim.load_state(*_state(np.full(n, e), np.outer(np.full(n, z), DIRECTION), phi=phi, pi=pi))
                sim.advance(1)
                got[math].append(sim.copy_state()[0][:, 1].astype(np.float64))
    return np.array(got["strict"]), np.array(got["fast"])


def _thermal_speed(eos_param, e, z, phi):
    """|v| of a cell in 64 bits, |Z| capped at 0.9999 E: bisection on the pressure."""
    gamma, a = eos_param
    z = min(z, 0.9999 * e)

    def excess(p):
        b, en = gamma * phi**2, e - z * z / (e + p)
        T = np.sqrt((0.5 * b + np.sqrt(0.25 * b * b + 0.5 * en)) / 0.25)
        return p - (0.125 / 3.0 * T**4 - 0.5 * b * T * T + a / 3.0 * T * phi**3)

    lo, hi = 0.0, 10.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if excess(mid) < 0.0 else (lo, mid)
    return z / (e + lo)


@pytest.mark.parametrize("eos_param", THERMAL)
def test_thermal_momentum_beyond_the_cap(bubble, gpu, eos_param):
    """Cold cells of the thermal potential have p > e, so |v| stays below the
    gamma = 3 threshold for |Z| beyond the cap.  Read through pi of uniform
    lattices, on which friction (W of v) and the thermal force (T) act and no
    flux.  Lattices of |v| < 0.8 when capped: the bar is then a hundred
    roundings of v (dW / dv <= 4; at W = 70, which capped warm cells reach, one
    rounding of v alone is 2e-2 of W)."""
    gamma, _ = eos_param
    branch = np.sqrt(3.0 * gamma / 0.5)
    states = []
    for T in (0.2, 0.26, 0.35, 0.5, 0.7, 1.0):
        for phi in (0.0, 0.3, 0.71, 1.0):
            if T >= 1.02 * branch * phi:
                e = _thermal_energy(gamma, T, phi)
                states += [(e, r * e, phi) for r in (0.0, 0.5, 0.9, 1.1, 1.27, 1.6)
                           if _thermal_speed(eos_param, e, r * e, phi) < 0.8]
    assert sum(z > e for e, z, _ in states) >= 3  # some beyond the cap
    strict, fast = _pi_after_a_step(bubble, states, eos_param, pi=0.01)
    err = np.max(np.abs(fast - strict), axis=1) / np.max(np.abs(strict), axis=1)
    assert np.all(err <= 1e-5), [(states[k], err[k]) for k in np.flatnonzero(err > 1e-5)]


@pytest.mark.parametrize("phi", [0.4, 1.0, 1.2])
def test_thermal_temperature_off_the_branch(bubble, gpu, phi):
    """With A < 1.5 gamma lo the phi = 0 root of the pressure solves p(T, phi) = p
    at T* = 2 A phi / (3 gamma), off the branch T >= lo phi, where the inversion
    must not stop.  Lattices at rest whose recovered T is T* within 3e-4; pi
    after a step is the thermal force at the inverted T."""
    gamma, a = 0.0208, 0.0095
    t_star = 2.0 * a * phi / (3.0 * gamma)
    assert np.sqrt(gamma / 0.25) * phi < t_star < np.sqrt(3.0 * gamma / 0.5) * phi
    states = [(_thermal_energy(gamma, t_star * (1.0 + d), phi), 0.0, phi) for d in np.linspace(-3e-4, 3e-4, 61)]
    strict, fast = _pi_after_a_step(bubble, states, (gamma, a), pi=0.0)
    err = np.max(np.abs(fast - strict), axis=1) / np.max(np.abs(strict), axis=1)
    assert np.all(err <= 1e-5), [(states[k], err[k]) for k in np.flatnonzero(err > 1e-5)]


@pytest.mark.parametrize("precision,eos,eos_param", [("single", "bag", (1.0, 0.0)), ("mixed", "bag", (1.0, 0.0)),
                                                     ("perturbation", "bag", (1.0, 0.0)),
                                                     ("single", "gamma_law", (1.2, 0.05)),
                                                     ("single", "thermal", (0.0125, 0.05))])
@pytest.mark.parametrize("component", range(6))
def test_nan_spreads_as_in_the_strict_form(bubble, gpu, component, precision, eos, eos_param):
    """A NaN in one component of a cell reaches the same values after a step,
    and the others are those of the strict form."""
    nx, ny, nz = GRID
    n = nx * ny * nz
    rng = np.random.default_rng(7)
    e = E_REF * rng.uniform(0.8, 1.2, n) - (E_REF if precision == "perturbation" else 0.0)
    f0, u0 = _state(e, E_REF * rng.uniform(-0.1, 0.1, (n, 3)), rng.uniform(-0.1, 1.1, n), rng.normal(0, 0.02, n))
    (f0 if component < 2 else u0)[(9 * ny + 10) * nx + 11, component % 4 if component < 2 else component - 2] = np.nan
    got = {}
    for math in ("strict", "fast"):
        spec = bubble.SimulationSpec(grid=GRID, bubbles=0, nucleation="centre", precision=precision, math=math, eos=eos,
                                     eos_param=eos_param)
        with bubble.Simulation(spec) as sim:
            sim.load_state(f0, u0)
            sim.advance(1)
            got[math] = np.concatenate(sim.copy_state(), axis=1).astype(np.float64)
    s, a = got["strict"], got["fast"]
    assert np.array_equal(np.isnan(a), np.isnan(s))
    err = np.nanmax(np.abs(a - s), axis=0) / np.nanmax(np.abs(s), axis=0)
    assert np.all(err <= 1e-5), err
