"""Chunks of a lattice served alone in the strict arithmetic.

On a fluid mostly at rest the strict kernel's items of one length differ up to
twofold in time, so a round of one long item per CTA waits for the slowest: 40
steps of 128^3 took 38.6 ms with such chunks and 27.4 with chunks of 6 planes.
The served time with the own pick is held to that of the set short chunk.
"""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu


def test_served_time_against_short_chunks(bubble, gpu):
    def served(chunk_planes):
        best = 1e9
        for _ in range(5):
            with bubble.Server(math="strict", chunk_planes=chunk_planes) as server:
                server.submit(bubble.SimulationSpec(grid=(128, 128, 128), bubbles=4, nucleation="simultaneous", seed=3,
                                                    math="strict"), 40)
                t = time.perf_counter()
                server.run_until_idle()
                best = min(best, time.perf_counter() - t)
        return best

    served(6)  # the first server of the process loads the kernels
    assert served(0) <= 1.15 * served(6)
