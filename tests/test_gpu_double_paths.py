"""The FP64 form on states that reach every branch of its comparisons.

The FP64 kernel compares doubles as integers and shares the velocity clamp
and the limiter's scaling between operations.  Random cells here have |Z| on
both sides of the cap z_max E, energies and pressures down to the floors,
equal neighbours (zero slopes) and slopes of both signs, at a spacing of 1
(where the divergence is not scaled) and another.  Both kernel paths, both
tiles and chunks of one plane, a remainder and the default are bit-identical
with the FP64 oracle.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(grid, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = grid
    n = nx * ny * nz
    field = np.stack([rng.normal(0.3, 0.3, n), rng.normal(0, 0.05, n)], 1)
    e = np.exp(rng.uniform(np.log(1e-3), 0, n))
    e[rng.random(n) < 0.03] = 1e-12  # below e_floor
    e[rng.random(n) < 0.3] = 0.125   # equal neighbours
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    speed = rng.choice([0.0, 0.3, 0.9, 0.99985, 0.9999, 1.2], size=n, p=[0.3, 0.3, 0.2, 0.08, 0.07, 0.05])
    return field, np.concatenate([e[:, None], d * (speed * e)[:, None]], 1)


@pytest.mark.parametrize("dx", [1.0, 0.7])
@pytest.mark.parametrize("grid", [(8, 8, 8), (17, 18, 9), (40, 21, 10)])
def test_double_bit_exact_on_extreme_states(bubble, oracle_mod, gpu, grid, dx):
    f0, u0 = _state(grid, 3)
    o = oracle_mod.OracleSim(grid, model=dict(oracle_mod.DEFAULT_MODEL, dx=dx), precision="f64")
    o.set_state(f0, u0)
    o.advance(1)
    fo, uo = o.state()
    assert np.isfinite(uo).all()
    spec = bubble.SimulationSpec(model=bubble.Model(dx=dx), grid=grid, bubbles=0, nucleation="centre", precision="double")
    for path, tile in (("fused", None), ("fused", (16, 1)), ("fused", (16, 4)), ("fused", (4, 5)), ("reference", None)):
        with bubble.Simulation(spec) as sim:
            sim.set_path(path)
            if tile:
                sim.set_tile(*tile)
            sim.load_state(f0, u0)
            sim.advance(1)
            f, u = sim.copy_state()
        assert np.array_equal(f, fo) and np.array_equal(u, uo), (path, tile)
