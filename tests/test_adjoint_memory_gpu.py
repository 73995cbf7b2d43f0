"""The loss and its gradient where device memory is short: a call whose
kernel-by-kernel form fits still runs, whatever the resident form would need."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(J1=-1.0, alpha=0.05, dt=0.005)


@pytest.mark.parametrize("states", [38, 42, 46, 60])
def test_loss_runs_in_what_the_plain_form_needs(states):
    """100 steps, checkpoints every 5: 36 state arrays kernel by kernel, 32 and a
    work space of 15 more in the resident form.  With room for `states` of them the
    call succeeds, again and again, and gives the gradient of a context that had all
    the memory it wanted."""
    N, nfile, steps, ckpt = 64, 100, 100, 5
    s0 = asd.random_spins(N, nfile, seed=3)
    target = np.full(10, 0.2 + 0.1j)
    p = asd.Params.make(N, nfile, **KW)
    with asd.Context(p, modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        want = ctx.loss_grad(steps, 10, ckpt, target)
    with asd.Context(p, modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        ctx.sqt("fp64")  # its work space
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        array = (N * N * nfile * 3 * 8 + (2 << 20) - 1) >> 21 << 21
        leave = states * array + (24 << 20)
        filler = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
        try:
            assert abs(torch.cuda.mem_get_info()[0] - leave) < array
            for _ in range(2):
                got = ctx.loss_grad(steps, 10, ckpt, target)
                assert abs(got[0] - want[0]) <= 1e-12 * want[0]
                assert np.abs(got[1] - want[1]).max() <= 1e-11 * np.abs(want[1]).max()
                assert np.abs(got[2] - want[2]).max() <= 1e-12
        finally:
            del filler
            torch.cuda.empty_cache()
