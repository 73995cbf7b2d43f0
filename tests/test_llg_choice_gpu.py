"""Sizes near the lines of the rule that picks the RK4 kernel: what the default takes
there, the measured faster one, and the stage kernels' spins bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,nfile,J2,nsteps,launches", [
    (32, 160, 0.0, 1, 1),     # resident 17.7 us, stage kernels 23.6
    (16, 600, 0.2, 1, 1),     # resident, up to 32 columns
    (64, 74, 0.0, 1, 4),      # stage kernels 29.9, resident 30 and more
    (80, 200, 0.2, 4, 16),    # stage kernels 422, resident 425
    (128, 150, 0.2, 2, 2),    # one-launch step 338, resident 346
    (128, 150, 0.2, 4, 1),    # resident 602, one-launch step 730
])
def test_default_near_a_line_of_the_rule(N, nfile, J2, nsteps, launches):
    s0 = asd.random_spins(N, nfile, seed=N)
    p = asd.Params.make(N, nfile, J1=-1.0, J2=J2, alpha=0.05, h=(0.0, 0.0, 0.5), dt=0.005)
    with asd.Context(p, modes=["fp64"]) as ctx:
        got = []
        for kernel in ("auto", "stages"):
            ctx.set_llg_kernel(kernel)
            ctx.set_spins(s0, as_origin=True)
            ctx.step(nsteps)
            if kernel == "auto":
                assert asd.load().asd_ctx_last_launches(ctx.handle) == launches
            got.append(ctx.get_spins())
    assert np.array_equal(*got)
