"""The FP64 q grid where the spins at t and at the origin differ in size: an error
of FP64 rounding in the product of the two, as with equal sizes."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


def reference(N, a, b):
    """S(q) and the scale of its rounding: the norms of the two operands."""
    def f(s):
        s = s.reshape(-1, N, N, 3)
        return np.fft.fft2(s - s.mean(axis=0), axes=(1, 2))

    A, B = f(a), f(b)
    norm = 1.0 / (N * N * len(a))
    return ((A * B.conj()).sum(axis=(0, 3)) * norm,
            np.sqrt((abs(A) ** 2).sum(axis=(0, 3)).max() * (abs(B) ** 2).sum(axis=(0, 3)).max())
            * norm)


@pytest.mark.parametrize("N,nfile", [(3, 2), (20, 16), (33, 7)])
@pytest.mark.parametrize("ratio", [1.0, 1.5, 1e8, 1e-8, 1e120, 1e-120])
def test_error_is_that_of_the_product(N, nfile, ratio):
    """The magnitudes are powers of ten apart, up to 1e120 (the product is in range).
    A transform of n points errs by about log2(n) eps of its norm, the sums add as
    much again: 8 log2(N^2) eps of the product of the norms."""
    b = asd.random_spins(N, nfile, seed=1)
    a = asd.random_spins(N, nfile, seed=2) * ratio
    want, scale = reference(N, a, b)
    with asd.Context(asd.Params.make(N, nfile), modes=["fp64"]) as ctx:
        ctx.set_spins(b, as_origin=True)
        for _ in range(2):
            ctx.set_spins(b, as_origin=False)
            ctx.sqt_grid("fp64")  # the size of an earlier state is forgotten
            ctx.set_spins(a, as_origin=False)
            got = ctx.sqt_grid("fp64")
            assert np.abs(got - want).max() <= 16 * np.log2(N) * 2.3e-16 * scale


def test_zero_and_huge_spins():
    N, nfile = 12, 4
    b = asd.random_spins(N, nfile, seed=1)
    with asd.Context(asd.Params.make(N, nfile), modes=["fp64"]) as ctx:
        ctx.set_spins(b, as_origin=True)
        ctx.set_spins(0.0 * b, as_origin=False)
        assert (ctx.sqt_grid("fp64") == 0.0).all()
        ctx.set_spins(b * 1e-200, as_origin=True)
        ctx.set_spins(b * 1e200, as_origin=False)
        got = ctx.sqt_grid("fp64")
        want, scale = reference(N, b, b)
        assert np.abs(got - want).max() <= 16 * np.log2(N) * 2.3e-16 * scale
        ctx.set_spins(b, as_origin=True)
        assert np.abs(ctx.sqt_grid("fp64") - want).max() <= 16 * np.log2(N) * 2.3e-16 * scale
