"""The chunk planner of the strict arithmetic's shared launches, on the CPU:
one cap for all lattices, the first of least cost."""
from __future__ import annotations

import os
import random
import subprocess

from conftest import PKG

MAIN = r"""
#include "chunk_plan.h"
#include <cstdio>
int main() {
    int max_grid, cap, n;
    while (scanf("%d %d %d", &max_grid, &cap, &n) == 3) {
        std::vector<bubble::ChunkPlanGrid> g(n);
        for (auto &x : g)
            if (scanf("%u %u %u", &x.nx, &x.ny, &x.nz) != 3) return 1;
        for (int v : bubble::spread_chunks(g, 16, 16, max_grid, cap)) printf("%d ", v);
        printf("\n");
    }
}
"""


def _cut(nz, cap):
    return -(-nz // -(-nz // cap))


def _expected(max_grid, cap_max, grids):
    def cost(cap):
        planes = sum(-(-x // 16) * -(-y // 16) * (z + 2 * -(-z // _cut(z, cap))) for x, y, z in grids)
        return planes / max_grid + max((_cut(z, cap) + 2 for _, _, z in grids), default=0)

    best, best_cap = 1e300, cap_max
    for cap in (cap_max, 48, 32, 24, 16, 12, 8, 6, 4):
        if cap <= cap_max and cost(cap) < best * (1 - 1e-9):
            best, best_cap = cost(cap), cap
    return [_cut(z, best_cap) for _, _, z in grids]


def test_spread_chunks(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "plan"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-I", str(PKG / "csrc"),
                    str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    rng = random.Random(2)
    cases = [(456, 64, []), (456, 64, [(128, 128, 128)]), (456, 3, [(40, 40, 40)])]
    for n in (1, 2, 5, 16):
        for lo, hi in ((8, 30), (30, 127)):
            cases.append((456, 64, [tuple(rng.randint(lo, hi) for _ in range(3)) for _ in range(n)]))
            cases.append((7, 200, [tuple(rng.randint(lo, hi) for _ in range(3)) for _ in range(n)]))
    text = "\n".join(f"{m} {c} {len(g)} " + " ".join(" ".join(map(str, x)) for x in g) for m, c, g in cases)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout
    got = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert got == [_expected(*c) for c in cases]
    assert got[1] == [6]  # 128^3 on 456 CTAs: short items
