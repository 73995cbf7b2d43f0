"""The q grid's device result at an address of eight bytes that is not one of
sixteen: the same values, and nothing written beside them."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mode", ["fp64", "tf32x3", "bf16x3", "fp16x3"])
@pytest.mark.parametrize("N,nfile", [(3, 1), (12, 5), (33, 20)])
def test_result_on_any_double_boundary(N, nfile, mode):
    n = 2 * N * N
    with asd.Context(asd.Params.make(N, nfile, alpha=0.1, dt=0.01), modes=[mode]) as ctx:
        ctx.set_spins(asd.random_spins(N, nfile, seed=N), as_origin=True)
        ctx.step(3)
        want = ctx.sqt_grid(mode)
        for shift in (0, 1):
            buf = torch.full((n + 3,), 7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ptr = buf.data_ptr() + 8 * shift
            assert ptr % 16 == 8 * shift
            ctx.sqt_grid_async(mode, ptr)
            ctx.synchronize()
            got = buf.cpu().numpy()
            assert np.array_equal(got[shift:shift + n].view(complex).reshape(N, N), want)
            assert (got[:shift] == 7.0).all() and (got[shift + n:] == 7.0).all()
