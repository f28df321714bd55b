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
