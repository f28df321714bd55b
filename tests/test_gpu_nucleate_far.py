"""Nucleation events whose centre lies far outside the lattice.

Events are the caller's; the profile is evaluated at the distance after one
fold by the lattice.  The cull that leaves bubbles out per brick must not lose
one whose wall just reaches a brick: thin walls (0.003 cells), centres and
radii of 1e7 cells whose wall lies on the last cell of a brick, and distances
whose square leaves the FP32 range.  Bit for bit against the oracle.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = (64, 16, 9)


@pytest.mark.parametrize("precision", ["single", "double"])
def test_bubble_wall_on_a_brick_edge(bubble, oracle_mod, gpu, precision):
    events = [(0.0, (1e7 + k, 4.0, 4.0), 1e7 + k - 64.0 - edge) for k in range(16) for edge in (31.0, 32.0)]
    events += [(0.0, (30.3, 7.7, 4.2), 6.1), (0.0, (-900.25, 3.0, 2.0), 880.0), (0.0, (3e20, 1.0, 1.0), 3.1e20),
               (0.0, (1e20, -2e20, 1.0), 1e25), (0.0, (4.0, 5.0, 6.0), 1e30)]
    kw = dict(lambda_=1e6)
    spec = bubble.SimulationSpec(grid=GRID, bubbles=0, nucleation="centre", precision=precision, model=bubble.Model(**kw))
    reached = 0
    with bubble.Simulation(spec) as sim:
        for ev in events:
            o = oracle_mod.OracleSim(GRID, model=dict(oracle_mod.DEFAULT_MODEL, **kw), schedule=[ev],
                                     precision="f64" if precision == "double" else "f32")
            o.record_nucleation()
            sim.reset([ev])
            sim.record_steps(0)
            f, f_ref = sim.copy_state()[0], o.state()[0]
            assert np.array_equal(f, f_ref), ev
            reached += bool((f_ref[:, 0] > 0).any())
    assert reached >= 32
