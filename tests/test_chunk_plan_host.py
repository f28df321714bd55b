"""The chunk planner of the shared launches, on the CPU.

The plan is the first of the shortest among all its candidates, simulated here
one by one, and finding it takes a small fraction of a round (it runs while
the GPU waits).
"""
from __future__ import annotations

import heapq
import os
import random
import subprocess

import pytest

from conftest import PKG

MAIN = r"""
#include "chunk_plan.h"
#include <chrono>
#include <cstdio>
// arguments on stdin: repeats, then per case: tx ty pair max_grid cap_max n, n x (nx ny nz)
int main() {
    int reps, tx, ty, pair, max_grid, cap, n;
    if (scanf("%d", &reps) != 1) return 1;
    while (scanf("%d %d %d %d %d %d", &tx, &ty, &pair, &max_grid, &cap, &n) == 6) {
        std::vector<bubble::ChunkPlanGrid> g(n);
        for (auto &x : g)
            if (scanf("%u %u %u", &x.nx, &x.ny, &x.nz) != 3) return 1;
        double best = 1e9;
        std::vector<int> lz;
        for (int r = 0; r < reps; ++r) {
            const auto t = std::chrono::steady_clock::now();
            lz = bubble::balanced_chunks(g, tx, ty, pair != 0, max_grid, cap);
            best = std::min(best, std::chrono::duration<double>(std::chrono::steady_clock::now() - t).count());
        }
        printf("%.9f", best);
        for (int v : lz) printf(" %d", v);
        printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def planner(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    exe = d / "plan"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-I", str(PKG / "csrc"), str(d / "main.cpp"), "-o",
                    str(exe)], check=True)

    def run(cases, reps=1):
        text = [str(reps)]
        for tx, ty, pair, max_grid, cap, grids in cases:
            text.append(f"{tx} {ty} {int(pair)} {max_grid} {cap} {len(grids)} " + " ".join(f"{a} {b} {c}" for a, b, c in grids))
        out = subprocess.run([str(exe)], input="\n".join(text), capture_output=True, text=True, check=True).stdout
        rows = [line.split() for line in out.splitlines()]
        return [float(r[0]) for r in rows], [[int(v) for v in r[1:]] for r in rows]

    return run


def _exhaustive(tx, ty, pair, max_grid, cap_max, grids):
    n, warm_up = len(grids), 1.6 if pair else 2.0

    def cut(nz, cap):
        return -(-nz // -(-nz // cap))

    def cost(lz):
        free, end, total = [0.0] * max_grid, 0.0, 0
        for (nx, ny, nz), z in zip(grids, lz):
            items = -(-nx // tx) * -(-ny // ty) * -(-nz // z)
            total += items
            for _ in range(items):
                t = heapq.heappop(free) + z + warm_up
                heapq.heappush(free, t)
                end = max(end, t)
        pace = 1.0 if not pair else 0.57 if 3 * total <= max_grid else 0.77 if 3 * total <= 2 * max_grid else 1.0
        return pace * end

    best, best_lz = 1e300, None
    caps = [cap_max] + [c for c in (48, 32, 24, 16, 12, 8, 6, 4) if c < cap_max]
    for k, a in enumerate(caps):
        plans = [(a, a, n)] + [(a, b, s) for b in caps[k + 1:] if b in (16, 8, 4) for s in (n // 4, n // 2, 3 * n // 4) if s]
        for first, rest, split in plans:
            lz = [cut(g[2], first if q < split else rest) for q, g in enumerate(grids)]
            c = cost(lz)
            if c < best * (1 - 1e-9):
                best, best_lz = c, lz
    return best_lz


def _grids(rng, n, lo, hi):
    g = [tuple(rng.randint(lo, hi) for _ in range(3)) for _ in range(n)]
    return sorted(g, key=lambda x: -x[0] * x[1] * x[2])


def test_plan_is_the_first_of_the_shortest(planner):
    rng = random.Random(3)
    cases = [(16, 16, True, 456, 64, [])]
    for n in (1, 2, 3, 7, 16):
        for lo, hi in ((8, 24), (32, 64), (8, 127)):
            cases.append((16, 16, True, 456, 64, _grids(rng, n, lo, hi)))
            cases.append((32, 8, False, 304, 1000, _grids(rng, n, lo, hi)))
            cases.append((16, 16, True, 7, 8, _grids(rng, n, lo, min(hi, 40))))
    cases.append((16, 16, True, 456, 64, [(128,) * 3] * 4 + [(96,) * 3] * 5 + [(64,) * 3] * 3 + [(48,) * 3] * 4))
    _, plans = planner(cases)
    assert plans == [_exhaustive(*c) or [] for c in cases]


def test_planning_is_short(planner):
    """64 lattices of different ragged sizes: 0.1 ms; 1.2 ms when every
    candidate is simulated to its end.  A round of such lattices takes 2 ms and
    more."""
    rng = random.Random(4)
    times, _ = planner([(16, 16, True, 456, 64, _grids(rng, 64, 8, 127)) for _ in range(4)], reps=20)
    assert max(times) < 0.6e-3, times
