"""The diagnostics pass on sizes and states where its shortcuts matter.

Lattices from the smallest to several items per block, odd in every axis, and
planes that are no multiple of a block; a fluid at rest, one whose momenta and
field fall from order one to subnormal (zero and tiny numerators take their own
way through the divisions), and one with |Z| beyond the cap.  Against the
oracle: FP64 sums within 1e-12 of the largest magnitude summed, max |v| and
the broken count exact.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(8, 8, 8), (33, 17, 10), (16, 16, 200), (97, 61, 75)]


def _state(grid, kind, e_ref, pert):
    n = grid[0] * grid[1] * grid[2]
    rng = np.random.default_rng(5)
    scale = np.ones(n)
    if kind == "rest":
        scale[:] = 0.0
    elif kind == "tails":
        scale = 10.0 ** rng.uniform(-45, 0, n)
        scale[rng.random(n) < 0.2] = 0.0
    field = np.stack([rng.uniform(-0.2, 1.2, n), rng.normal(0, 0.1, n)], 1) * scale[:, None]
    de = 0.05 * rng.uniform(-1, 1, n) * scale
    e = e_ref + de
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    speed = rng.choice([0.1, 0.6, 0.97, 0.99985, 1.1], size=n) if kind == "capped" else rng.uniform(0, 0.6, n)
    z = d * (speed * e * scale)[:, None]
    return field.astype(np.float32), np.concatenate([(de if pert else e)[:, None], z], 1).astype(np.float32)


@pytest.mark.parametrize("precision", ["single", "mixed", "perturbation"])
@pytest.mark.parametrize("kind", ["rest", "tails", "capped"])
@pytest.mark.parametrize("grid", GRIDS)
def test_diagnostics_match_oracle(bubble, oracle_mod, gpu, grid, kind, precision):
    o = oracle_mod.OracleSim(grid, precision={"single": "f32", "mixed": "mixed", "perturbation": "pert"}[precision])
    f0, u0 = _state(grid, kind, float(o.d["e_ref"]), precision == "perturbation")
    o.set_state(f0, u0)
    ref = o.diagnostics()
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", precision=precision)
    with bubble.Simulation(spec) as sim:
        sim.load_state(f0, u0)
        d, again = sim.diagnostics(), sim.diagnostics()
    for k in ("sum_energy", "sum_kinetic", "sum_fluid_energy"):
        big = max(abs(ref[k]), 1e-30)
        assert abs(getattr(d, k) - ref[k]) <= 1e-12 * big, (k, getattr(d, k), ref[k])
    assert d.sum_broken == ref["sum_broken"]
    assert np.float32(d.max_velocity) == np.float32(ref["max_velocity"])
    assert d == again
