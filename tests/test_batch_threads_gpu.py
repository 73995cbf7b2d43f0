"""Spins of a batch set and read by several threads at once, each its own lattices."""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


def test_threads_set_and_get_their_own_lattices():
    sides = [96 + 8 * (l % 9) for l in range(32)]
    spins = [asd.random_spins(n, 1, seed=l)[0].astype(np.float32) for l, n in enumerate(sides)]
    with asd.Batch([asd.Lattice.make(n) for n in sides]) as b, ThreadPoolExecutor(8) as pool:
        for _ in range(20):
            list(pool.map(lambda l: b.set_spins(l, spins[l]), range(len(sides))))
            got = list(pool.map(b.get_spins, range(len(sides))))
            for x, y in zip(got, spins):
                assert np.array_equal(x, y)
