"""The pair form of the fused stage kernel (fast bag forms, 16 x 16 tiles).

Sizes where its layout can go wrong: the smallest lattice, one tile exactly,
tiles that reach past the lattice by a row, by all but one, or in x only, rows
on both halves of a pair, the smallest lattices with a TMA-staged tile, and z
chunks of one plane, of a remainder and of the whole column.  Every chunking
gives the same bits.  Accuracy is that of the strict FP32 form: per component
(largest error over largest magnitude) against the FP64 form after two steps,
no more than 2 err(strict) + 1e-6, the bar of the MIXED form's own test; the
two are separate roundings of one scheme, so their errors agree in size and
not cell by cell.
"""
from __future__ import annotations

import numpy as np
import pytest

import make_golden

pytestmark = pytest.mark.gpu

GRIDS = [(8, 8, 8), (16, 16, 16), (17, 9, 10), (33, 31, 8), (15, 25, 12), (36, 34, 9), (50, 48, 20)]
STEPS = 2


def _state(oracle_mod, grid, kind):
    sched = oracle_mod.make_schedule("centre", 1, 4.0, grid, 10.0, 1)
    o = oracle_mod.OracleSim(grid, schedule=sched, precision="f32")
    o.advance(2)
    if kind == "mixed":  # cells above gamma = 3 beside cells below it
        make_golden.relativistic_state(o, 5, 0.99)
    else:
        make_golden.perturbed_state(o, 5, 0.3)
    f, u = o.state()
    return f, u, float(o.d["e_ref"])


def _run(bubble, grid, f0, u0, precision, math, lz=None, **kw):
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", precision=precision, math=math, **kw)
    with bubble.Simulation(spec) as sim:
        if lz is not None:
            sim.set_tile(16, lz)
        sim.load_state(f0, u0)
        sim.advance(STEPS)
        return sim.copy_state()


def _err(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    scale = np.max(np.abs(b), axis=0)
    scale[scale == 0] = 1.0
    return np.max(np.abs(a - b), axis=0) / scale


@pytest.mark.parametrize("precision", ["single", "mixed", "perturbation"])
@pytest.mark.parametrize("grid", GRIDS)
def test_pair_form(bubble, oracle_mod, gpu, grid, precision):
    f0, u0, e_ref = _state(oracle_mod, grid, precision)
    f64, u64 = f0.astype(np.float64), u0.astype(np.float64)
    shift = np.zeros(4)
    if precision == "perturbation":  # stored form: E - e_ref
        u0 = u0.copy()
        u0[:, 0] = (u0[:, 0] - np.float32(e_ref)).astype(np.float32)
        u64 = u0.astype(np.float64) + [e_ref, 0, 0, 0]
        shift = np.array([e_ref, 0, 0, 0])
    ref = _run(bubble, grid, f64, u64, "double", "strict")
    strict = _run(bubble, grid, f0, u0, precision, "strict")
    fast = _run(bubble, grid, f0, u0, precision, "fast")
    for a, s, r, off in ((fast[0], strict[0], ref[0], np.zeros(2)), (fast[1], strict[1], ref[1], shift)):
        e_fast, e_strict = _err(a, r - off), _err(s, r - off)
        assert np.all(e_fast <= 2.0 * e_strict + 1e-6), (e_fast, e_strict)
    for lz in (1, 3, grid[2]):
        got = _run(bubble, grid, f0, u0, precision, "fast", lz)
        assert np.array_equal(got[0], fast[0]) and np.array_equal(got[1], fast[1]), lz


E_REF = 0.125  # e_ref = a_rad of the default model
EOS = [("gamma_law", (1.2, 0.05)), ("gamma_law", (2.0, 0.0)), ("gamma_law", (1.02, 0.12)), ("thermal", (0.0, 0.0)),
       ("thermal", (0.0125, 0.05)), ("thermal", (0.999 * E_REF / 6.0, 0.999 * E_REF / np.sqrt(2.0)))]


@pytest.mark.parametrize("eos,eos_param", EOS)
@pytest.mark.parametrize("grid", GRIDS)
def test_pair_form_other_equations_of_state(bubble, oracle_mod, gpu, grid, eos, eos_param):
    """The gamma law's closed-form recovery and the thermal potential's short
    iterations against the strict form's eight Newton steps: the fast
    arithmetic's bar of 1e-5 per component, and the same bits for every
    chunking."""
    f0, u0, _ = _state(oracle_mod, grid, "single")
    kw = dict(eos=eos, eos_param=eos_param)
    strict = _run(bubble, grid, f0, u0, "single", "strict", **kw)
    fast = _run(bubble, grid, f0, u0, "single", "fast", **kw)
    for a, s in zip(fast, strict):
        assert np.isfinite(a).all() and np.all(_err(a, s) <= 1e-5), _err(a, s)
    for lz in (1, 3, grid[2]):
        got = _run(bubble, grid, f0, u0, "single", "fast", lz, **kw)
        assert np.array_equal(got[0], fast[0]) and np.array_equal(got[1], fast[1]), lz


@pytest.mark.parametrize("precision", ["single", "mixed", "perturbation"])
def test_combine_keeps_small_increments(bubble, gpu, precision):
    """Where a step changes E and Z by about an ulp, the order of the stage
    combine decides which increments are dropped: after 100 steps the root mean
    square error against the FP64 form is that of the strict form, and double
    when the last stage drops those below 3/4 ulp.  The bar lies between."""
    kw = dict(grid=(96, 96, 96), nucleation="simultaneous", bubbles=4, seed=1)

    def run(precision, math):
        with bubble.Simulation(bubble.SimulationSpec(precision=precision, math=math, **kw)) as sim:
            sim.advance(100)
            field, fluid = sim.copy_state()
            return np.asarray(field, np.float64), np.asarray(fluid, np.float64)

    ref, strict, fast = run("double", "strict"), run(precision, "strict"), run(precision, "fast")
    if precision == "perturbation":  # stored form: E - e_ref
        ref[1][:, 0] -= E_REF
    for a, s, r in ((fast[0], strict[0], ref[0]), (fast[1], strict[1], ref[1])):
        e_fast, e_strict = np.linalg.norm(a - r, axis=0), np.linalg.norm(s - r, axis=0)
        assert np.all(e_fast <= 1.5 * e_strict), (e_fast, e_strict)


@pytest.mark.parametrize("precision,math", [("mixed", "fast"), ("single", "strict")])
def test_step_under_capture(bubble, oracle_mod, gpu, precision, math):
    """A step recorded into a CUDA graph (plain launches there, dependent ones
    outside) and replayed gives the bits of a step launched directly."""
    import torch

    grid = (50, 48, 20)
    f0, u0, _ = _state(oracle_mod, grid, "single")
    spec = bubble.SimulationSpec(grid=grid, bubbles=0, nucleation="centre", precision=precision, math=math)
    with bubble.Simulation(spec) as sim:
        sim.load_state(f0, u0)
        sim.advance(2)
        want = sim.copy_state()
    stream = torch.cuda.Stream()
    with bubble.Simulation(spec) as sim:
        sim.set_stream(stream.cuda_stream)
        sim.load_state(f0, u0)
        sim.advance(1)
        sim.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sim.record_steps(1)
        graph.replay()
        torch.cuda.synchronize()
        got = sim.copy_state()
        sim.set_stream(None)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
