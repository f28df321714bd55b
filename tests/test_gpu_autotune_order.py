"""The chunk autotuner's memory: what a batch timed (chunks of 4 planes and
more, all that its creation waits for) does not stand in for the short chunks
of a lattice by itself, and the other way round."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu


def _batch(bubble, n):
    spec = bubble.SimulationSpec(grid=(n, n, n), bubbles=1, nucleation="centre")
    t = time.perf_counter()
    with bubble.Batch([spec]) as batch:
        t = time.perf_counter() - t
        batch.advance(2)
        return t, batch.copy_state(0)


def test_batch_and_single_picks_are_separate(bubble, gpu):
    _batch(bubble, 24)  # loads the kernels
    first, a = _batch(bubble, 36)
    assert 1 <= bubble.autotune_chunk((36, 36, 36), 16, "fast") <= 3
    again, b = _batch(bubble, 36)
    assert 1 <= bubble.autotune_chunk((36, 36, 36), 16, "fast") <= 3
    assert all((x == y).all() for x, y in zip(a, b))
    # a tuned single lattice leaves the batch of that size nothing to time
    assert 1 <= bubble.autotune_chunk((44, 44, 44), 16, "fast") <= 3
    tuned, _ = _batch(bubble, 44)
    untuned, _ = _batch(bubble, 40)
    assert tuned < untuned
