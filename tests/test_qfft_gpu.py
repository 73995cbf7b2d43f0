"""S(q,t) on the whole q grid in FP64 (2-D transforms of the spins) against
numpy's FFT of the same spins, over the lattice sides whose factors take each
path of the transform (radix 8, 4, 2, 3, 5, other primes, several of them), and
replica counts that leave a part of a block of 8 columns; a second q-grid call
gives the same bits.

Tolerance: log2(M) <= 14 rounding steps of 2^-53 per value, K sums; 1e-12 of the
largest |S(q)|, the bound of the FP64 grid in the other tests."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


def numpy_grid(N, nf, st, s0):
    A = np.fft.fft2((st - st.mean(axis=0)).reshape(nf, N, N, 3), axes=(1, 2))
    B = np.fft.fft2((s0 - s0.mean(axis=0)).reshape(nf, N, N, 3), axes=(1, 2))
    return (A * B.conj()).sum(axis=(0, 3)) / (N * N * nf)


@pytest.mark.parametrize("N,nfile", [(3, 2), (4, 5), (5, 3), (7, 8), (8, 11), (13, 3), (16, 86),
                                     (30, 4), (49, 2), (51, 7), (64, 9), (67, 3), (96, 5), (121, 2),
                                     (125, 3), (128, 40), (256, 3), (600, 2), (601, 2), (1024, 2),
                                     (2432, 1)])
def test_fp64_grid_over_the_transform_paths(N, nfile):
    s0 = asd.random_spins(N, nfile, seed=11 * N + nfile)
    with asd.Context(asd.Params.make(N, nfile, J1=1.0, alpha=0.1, dt=0.01), modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.step(2)
        st = ctx.get_spins()
        got = ctx.sqt_grid("fp64")
        again = ctx.sqt_grid("fp64")
    want = numpy_grid(N, nfile, st, s0)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    assert np.array_equal(got, again)


def test_chunks_of_columns_add_up():
    """200 x 200 with 60 replicas: 180 columns in chunks of 72, 72 and 36."""
    N, nfile = 200, 60
    s0 = asd.random_spins(N, nfile, seed=1)
    with asd.Context(asd.Params.make(N, nfile, J1=-1.0, dt=0.01), modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.step(1)
        st = ctx.get_spins()
        got = ctx.sqt_grid("fp64")
    want = numpy_grid(N, nfile, st, s0)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()


def test_one_replica_has_no_connected_part():
    with asd.Context(asd.Params.make(24, 1, J1=1.0, dt=0.01), modes=["fp64"]) as ctx:
        ctx.set_spins(asd.random_spins(24, 1, seed=2), as_origin=True)
        ctx.step(3)
        assert np.abs(ctx.sqt_grid("fp64")).max() == 0.0
