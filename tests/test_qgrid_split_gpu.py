"""The split-mode q grid against the FP64 one where its epilogue's index sets can
go wrong: lattice sides below, at and past the 32 columns of a block (a class
boundary in every block, in one or in none), sides that leave ragged tiles,
several tiles a CTA and several chunks of K; a second call gives the same bits.

Tolerance: 1e-5 of the largest |S(q)|, the split modes' bound elsewhere."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nfile", [(3, 2), (5, 3), (12, 100), (31, 9), (32, 100), (33, 9),
                                     (63, 5), (97, 20), (128, 3)])
def test_split_grid_matches_fp64(N, nfile):
    s0 = asd.random_spins(N, nfile, seed=7 * N + nfile)
    with asd.Context(asd.Params.make(N, nfile, J1=1.0, alpha=0.1, dt=0.01)) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.step(2)
        want = ctx.sqt_grid("fp64")
        for mode in ("tf32x3", "bf16x3", "fp16x3"):
            got = ctx.sqt_grid(mode)
            assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), mode
            assert np.array_equal(got, ctx.sqt_grid(mode)), mode
