"""The split-mode q grid's sums over a tile, its K chunks and its warps hold what
FP64 holds: no overflow where every value summed is finite in FP32, and the value of
the FP64 grid to the accuracy of the split operands at any size of the spins."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu

MODES = ("tf32x3", "bf16x3", "fp16x3")


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("N,nfile,chunk", [(16, 2, -1), (20, 2, -1), (16, 256, 128)])
def test_sums_of_finite_values_stay_finite(N, nfile, chunk, mode):
    """Half of the replicas +s, half -s along z at every site: every value is s^2, 32
    of them are finite in FP32 and 128, a tile's longest diagonal, are not."""
    s = 2.0 ** 61
    spins = np.zeros((nfile, N * N, 3))
    spins[: nfile // 2, :, 2], spins[nfile // 2:, :, 2] = s, -s
    with asd.Context(asd.Params.make(N, nfile, spin_len=s), modes=[mode]) as ctx:
        ctx.set_chunk_k(chunk)
        ctx.set_spins(spins, as_origin=True)
        got = ctx.sqt_grid(mode)
    want = np.zeros((N, N), dtype=complex)
    want[0, 0] = N * N * s * s
    assert np.abs(got - want).max() <= 1e-6 * want[0, 0].real


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("N,nfile,chunk", [(33, 10, -1), (33, 300, 128), (20, 90, 64)])
def test_any_power_of_two_scales_the_grid(N, nfile, chunk, mode):
    """Spins times 2^k give the grid times 2^2k exactly, from 2^-40 to 2^57 (the
    largest the operands' FP32 products hold), whatever size is near the limits."""
    spins = asd.random_spins(N, nfile, seed=N)
    got = {}
    for k in (0, -40, 30, 52, 57):
        f = 2.0 ** k
        with asd.Context(asd.Params.make(N, nfile, spin_len=f), modes=[mode]) as ctx:
            ctx.set_chunk_k(chunk)
            ctx.set_spins(spins * f, as_origin=True)
            got[k] = ctx.sqt_grid(mode) / f / f
    assert np.abs(got[0]).max() > 0.1
    for k, v in got.items():
        assert np.array_equal(v, got[0]), k
