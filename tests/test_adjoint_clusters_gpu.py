"""The resident adjoint with one, two and four CTAs a replica, on lattice sides whose
rows do not divide among them, against the kernel-by-kernel adjoint: two CTAs are each
other's neighbour both above and below, four have one each.

Tolerance: rounding only, some hundred operations a step over 11 steps on values of
order one; 1e-11 of the largest component."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu

MODELS = [dict(J1=1.0, dt=0.02), dict(J1=-1.0, alpha=0.05, h=(0.1, -0.2, 0.5), dt=0.01),
          dict(J1=0.8, J2=0.2, alpha=0.15, dt=0.01), dict(J1=-1.0, J2=-0.3, dt=0.01)]


def with_ctas(N, ctas):
    """A number of replicas for which the default takes `ctas` CTAs a replica."""
    for nfile in (70, 74, 50, 60, 66, 40, 30, 16, 100, 148, 200):
        if asd.load().asd_check_adjoint_ctas(N, nfile, 148) == ctas:
            return nfile
    raise AssertionError((N, ctas))


@pytest.mark.parametrize("model", range(len(MODELS)))
@pytest.mark.parametrize("N,ctas", [(13, 1), (19, 1), (31, 1), (33, 2), (35, 2), (51, 2), (62, 2),
                                    (63, 2), (64, 2), (33, 4), (35, 4), (49, 4), (62, 4), (63, 4)])
def test_every_cluster_size_equals_the_kernel_by_kernel_adjoint(N, ctas, model):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the replica counts are chosen for 148 SMs")
    nfile = with_ctas(N, ctas)
    s0 = asd.random_spins(N, nfile, seed=N)
    target = (0.9 ** np.arange(1, 6)) * (1.0 + 0.1j)
    out = []
    p = asd.Params.make(N, nfile, vx=1, vy=2, **MODELS[model])
    with asd.Context(p, modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        for kernel in ("stages", "auto"):
            ctx.set_llg_kernel(kernel)
            f = ctx.loss_forward(11, 2, 4, target)
            g, _ = ctx.loss_backward(target)
            out.append((f[0], f[1], g, ctx.last_launches()))
    a, b = out
    assert b[3] <= 3 + 1  # one per segment and the final sum
    np.testing.assert_allclose(b[1], a[1], rtol=1e-13, atol=1e-15)
    assert abs(b[0] - a[0]) <= 1e-13 * abs(a[0])
    assert np.abs(b[2] - a[2]).max() <= 1e-11 * np.abs(a[2]).max(), (a[2], b[2])
