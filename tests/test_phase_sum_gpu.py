"""S(q,t) at one q in FP64 (column sums over the sites, their products with the
origin's) against the oracle's factorised long-double form, at the edges of the
kernels: one and two columns per thread (odd and even K = 3 nfile), a last block
of columns with one thread's worth, chunks of rows with a remainder, one replica.

Tolerance: each column sum is a chain of at most 256 fused multiply-adds and one
of at most M / 16 / 8 chunk sums, so its rounding is below (256 + M / 128 + 8)
2^-53 of the sum of its terms' magnitudes; random signs keep the rest far below.
1e-12 of |S| plus 1e-15 for the sizes where S is (near) zero."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nfile", [(3, 1), (3, 2), (17, 43), (16, 86), (33, 11), (64, 171),
                                     (65, 170), (100, 3)])
def test_column_sums_at_block_and_chunk_edges(oracle, N, nfile):
    s0 = asd.random_spins(N, nfile, seed=7 * N + nfile)
    kw = dict(J1=1.0, alpha=0.1, dt=0.01)
    with asd.Context(asd.Params.make(N, nfile, vx=1, vy=2, **kw), modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.step(2)
        st = ctx.get_spins()
        got = ctx.sqt("fp64")
        want = oracle.sqt_factorized(N, nfile, 1, 2, st, s0)
        assert abs(got - want) <= 1e-12 * abs(want) + 1e-15, (got, want)
        assert ctx.sqt("fp64") == got
        # another q, then another origin: the origin's sums are formed again
        ctx.set_params(asd.Params.make(N, nfile, vx=2, vy=0, **kw))
        want = oracle.sqt_factorized(N, nfile, 2, 0, st, s0)
        assert abs(ctx.sqt("fp64") - want) <= 1e-12 * abs(want) + 1e-15
        s1 = asd.random_spins(N, nfile, seed=7 * N + nfile + 1)
        ctx.set_spins(s1, as_origin=True)
        ctx.set_spins(st)
        want = oracle.sqt_factorized(N, nfile, 2, 0, st, s1)
        assert abs(ctx.sqt("fp64") - want) <= 1e-12 * abs(want) + 1e-14, (ctx.sqt("fp64"), want)
