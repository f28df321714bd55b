"""The z chunk that the fused kernel's launches march.

Each arithmetic picks the cheapest chunk of its own cost model (restated here
for a cube), a chunk that was set is the one that runs, and setting the tile
that is reported changes nothing.  Any chunk gives the same bits.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _pair_cost(n, lz, sms):
    tiles, chunks = ((n + 15) // 16) ** 2, -(-n // lz)
    ctas = tiles * chunks
    m = -(-ctas // sms)
    full = (m - 1) // 3
    rounds = full + {1: 0.57, 2: 0.77, 3: 1.0}[m - 3 * full]
    share = ctas / (3.0 * sms)
    waves = rounds if share <= 1.0 else 0.8 * rounds + 0.2 * share
    return waves * (-(-n // chunks) + 1.6) + 0.64


def _fp64_cost(n, lz, sms):
    tiles = ((n + 15) // 16) ** 2
    a, b = lz + 0.73, n % lz + 0.73
    full, rest = tiles * (n // lz), tiles if n % lz else 0
    m, x = divmod(full, sms)
    cost = (m + 1 if x else m) * a
    room = (sms - x) * int(a / b) if x else 0
    return cost if rest <= room else cost + -(-(rest - room) // sms) * b


def _spec(bubble, n, **kw):
    return bubble.SimulationSpec(grid=(n, n, n), bubbles=1, nucleation="centre", **kw)


@pytest.mark.parametrize("n", [8, 32, 64, 97, 128, 256])
@pytest.mark.parametrize("kw,cost", [(dict(), _pair_cost), (dict(precision="mixed"), _pair_cost),
                                     (dict(precision="double"), _fp64_cost)], ids=["single", "mixed", "double"])
def test_default_chunk_is_the_cheapest(bubble, gpu, n, kw, cost):
    if n == 256 and "double" in kw.values():
        n = 160
    sms = _sms()
    with bubble.Simulation(_spec(bubble, n, **kw)) as sim:
        lz = sim.chunk()
    assert 1 <= lz <= n
    assert cost(n, lz, sms) <= min(cost(n, k, sms) for k in range(1, n + 1)) * (1 + 1e-6)


@pytest.mark.parametrize("n", [32, 48, 96, 160])
def test_setting_the_reported_tile_changes_nothing(bubble, gpu, n):
    with bubble.Simulation(_spec(bubble, n)) as sim:
        pick = sim.chunk()
        tile = sim.tile()
        sim.set_tile(*tile)
        assert (sim.chunk(), sim.tile()) == (pick, tile)
        sim.set_tile(16, 3)
        assert (sim.chunk(), sim.tile()) == (3, (16, 3))
        sim.set_tile(8, 7)
        assert (sim.chunk(), sim.tile()) == (7, (8, 7))
        sim.set_tile(*tile)
        assert (sim.chunk(), sim.tile()) == (pick, tile)
        sim.resize((64, 64, 64))
        assert sim.chunk() == _fresh_chunk(bubble, 64)
    with bubble.Simulation(_spec(bubble, n, math="strict")) as sim:
        assert sim.chunk() == sim.tile()[1]
        sim.set_tile(16, 3)
        assert sim.chunk() == 3


def _fresh_chunk(bubble, n):
    with bubble.Simulation(_spec(bubble, n)) as sim:
        return sim.chunk()


@pytest.mark.parametrize("precision", ["single", "mixed", "perturbation"])
def test_default_chunk_at_128_cubed(bubble, oracle_mod, gpu, precision):
    """The fast arithmetic's own pick against a set chunk, and the strict
    register and shared forms against each other, where tiles are TMA-staged and
    chunks end unevenly."""
    kw = dict(grid=(128, 128, 128), bubbles=4, nucleation="simultaneous", seed=3, precision=precision)

    def run(form=None, lz=None, **more):
        with bubble.Simulation(bubble.SimulationSpec(**kw, **more)) as sim:
            if form:
                sim.set_stage_form(form)
            if lz:
                sim.set_tile(16, lz)
            used = sim.chunk()
            sim.advance(4)
            return used, *sim.copy_state()

    used, *auto = run()
    for lz in (used + 1, 32, 128):
        got = run(lz=lz)
        assert got[0] == lz
        assert np.array_equal(got[1], auto[0]) and np.array_equal(got[2], auto[1]), lz
    _, *regs = run("registers", 32, math="strict")
    _, *shared = run("shared", 19, math="strict")
    assert np.array_equal(regs[0], shared[0]) and np.array_equal(regs[1], shared[1])


@pytest.mark.parametrize("n", [32, 40, 48])
def test_autotuner_finds_the_short_chunks(bubble, gpu, n):
    """On small lattices the pair form's best chunk is 1 or 2 planes, 1.3 to 1.7
    times as fast as any of 4 and more; a tuned chunk that is set runs."""
    lz = bubble.autotune_chunk((n, n, n), 16, "fast")
    assert 1 <= lz <= 3
    with bubble.Simulation(_spec(bubble, n)) as sim:
        sim.set_tile(16, lz)
        assert sim.chunk() == lz
