"""Chunk plans of the shared launches (the request loop).

A round's lattices are cut by a plan that depends on which lattices share it:
one cap, or a smaller one for the smaller lattices.  Whatever the plan, a
lattice's bits are those of the same lattice alone.  Mixes where the plan can
go wrong: one lattice, equal lattices (one run of items), as many distinct
ragged sizes as lattices, more items than CTAs, and a configured cap below
every candidate.
"""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu

MIXES = {
    "one": [(48, 48, 48)],
    "equal": [(32, 32, 32)] * 5,
    "ragged": [(97, 61, 40), (50, 48, 20), (33, 31, 8), (17, 9, 70), (8, 8, 8), (64, 40, 33)],
    "many": [(96, 96, 96)] * 4 + [(64, 64, 64)] * 3 + [(48, 48, 48)] * 3 + [(32, 32, 32)],
}


def _specs(bubble, mix, math):
    return [bubble.SimulationSpec(grid=g, nucleation="centre", bubbles=1, math=math) for g in MIXES[mix]]


def _sums(d):
    return [d.sum_energy, d.sum_broken, d.sum_kinetic, d.sum_fluid_energy, d.max_velocity]


@pytest.mark.parametrize("math,tile_y", [("fast", 16), ("strict", 16), ("fast", 8)])
@pytest.mark.parametrize("mix", MIXES)
def test_served_alone_and_together(bubble, gpu, mix, math, tile_y):
    specs = _specs(bubble, mix, math)
    steps = [3 + 2 * (k % 4) for k in range(len(specs))]
    alone = []
    with bubble.Server(math=math, tile_y=tile_y) as server:
        for spec, n in zip(specs, steps):
            server.submit(spec, n)
            server.run_until_idle()
            alone += [_sums(r["diag"]) for r in server.poll()]
    for planes in (0, 2, 1000):
        with bubble.Server(math=math, tile_y=tile_y, chunk_planes=planes) as server:
            ids = [server.submit(spec, n) for spec, n in zip(specs, steps)]
            server.run_until_idle()
            got = {r["id"]: _sums(r["diag"]) for r in server.poll()}
        assert [got[i] for i in ids] == alone, planes
