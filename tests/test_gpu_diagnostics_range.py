"""Reports of states whose terms leave the FP32 range.

The report sums FP32 terms over chunks of planes in FP32 pairs; where such a
sum overflows, or a term is infinite or NaN, it is the sum in FP64 of the same
terms all the same: finite where that is finite, infinite where that is.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["single", "mixed", "perturbation"])
@pytest.mark.parametrize("kind", ["huge", "infinite", "nan"])
@pytest.mark.parametrize("grid", [(8, 8, 8), (97, 61, 75)])
def test_sums_beyond_the_fp32_range(bubble, oracle_mod, gpu, grid, kind, precision):
    nx, ny, nz = grid
    o = oracle_mod.OracleSim(grid, precision={"single": "f32", "mixed": "mixed", "perturbation": "pert"}[precision])
    rng = np.random.default_rng(4)
    field = rng.normal(0, 0.1, (nz, ny, nx, 2)).astype(np.float32)
    fluid = np.zeros((nz, ny, nx, 4), np.float32)
    fluid[..., 0] = 0.125 * rng.uniform(0.9, 1.1, (nz, ny, nx)) - (0.125 if precision == "perturbation" else 0.0)
    if kind == "huge":  # a column of cells whose energies overflow FP32 together
        fluid[:, 3, 5, 0] = 3e38
    else:
        fluid[nz // 2, 3, 5, 0] = {"infinite": np.inf, "nan": np.nan}[kind]
        field[1, 2, 7, 1] = np.inf
    f0, u0 = field.reshape(-1, 2), fluid.reshape(-1, 4)
    o.set_state(f0, u0)
    ref = o.diagnostics()
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", precision=precision)
    with bubble.Simulation(spec) as sim:
        sim.load_state(f0, u0)
        d = sim.diagnostics(allow_nonfinite=True)
    for k in ("sum_energy", "sum_kinetic", "sum_fluid_energy", "sum_broken"):
        np.testing.assert_allclose(getattr(d, k), ref[k], rtol=1e-12, atol=0, err_msg=k)
