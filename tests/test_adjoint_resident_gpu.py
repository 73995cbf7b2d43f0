"""The resident adjoint (a segment's backward pass in one launch, a replica's
lattice on one or two SMs; the default from 16 replicas on) against the
kernel-by-kernel adjoint on the same inputs: loss and S(q,t) equal, gradients
equal up to the order and contraction of FP64 sums.  Sizes at the edges of its
geometry (one CTA and two per replica, idle threads, uneven halves, the smallest
and largest lattice side), every combination of the model's terms, segments that
do and do not divide the steps, a segment of one step, and evaluations that do
not fall on every step.

Tolerance: the two differ in rounding only, some hundred operations a step over at
most 20 steps on values of order one; 1e-11 of the largest component leaves four
digits to spare."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu

MODELS = [dict(J1=1.0, dt=0.02), dict(J1=-1.0, alpha=0.05, h=(0.1, -0.2, 0.5), dt=0.01),
          dict(J1=0.8, J2=0.2, alpha=0.15, dt=0.01), dict(J1=-1.0, J2=-0.3, dt=0.01)]


def gradients(N, nfile, kw, nsteps, stride, ckpt):
    s0 = asd.random_spins(N, nfile, seed=N * 5 + nfile)
    E = nsteps // stride
    target = (0.9 ** np.arange(1, E + 1)) * (1.0 + 0.1j)
    out = []
    with asd.Context(asd.Params.make(N, nfile, vx=1, vy=2, **kw), modes=["fp64"]) as ctx:
        ctx.set_spins(s0, as_origin=True)
        for kern in ("stages", "auto"):
            ctx.set_llg_kernel(kern)
            out.append(ctx.loss_grad(nsteps, stride, ckpt, target))
            ctx.set_llg_kernel(kern)
            f = ctx.loss_forward(nsteps, stride, ckpt, target)
            g, _ = ctx.loss_backward(target)
            launches = ctx.last_launches()
            assert f[0] == out[-1][0] and np.array_equal(g, out[-1][1])
    return out, launches


@pytest.mark.parametrize("model", range(len(MODELS)))
@pytest.mark.parametrize("N", [12, 13, 17, 32, 33, 34, 51, 63, 64])
def test_equals_the_kernel_by_kernel_adjoint(N, model):
    nsteps, stride, ckpt = 11, 2, 4
    (a, b), launches = gradients(N, 18, MODELS[model], nsteps, stride, ckpt)
    assert launches <= 3 + 1  # one per segment and the final sum
    np.testing.assert_allclose(b[2], a[2], rtol=1e-13, atol=1e-15)
    assert abs(b[0] - a[0]) <= 1e-13 * abs(a[0])
    assert np.abs(b[1] - a[1]).max() <= 1e-11 * np.abs(a[1]).max(), (a[1], b[1])


@pytest.mark.parametrize("nsteps,stride,ckpt", [(1, 1, 1), (5, 5, 1), (6, 1, 6), (7, 3, 50), (20, 7, 3)])
def test_segments_and_strides(nsteps, stride, ckpt):
    (a, b), _ = gradients(20, 160, MODELS[1], nsteps, stride, ckpt)
    assert np.abs(b[1] - a[1]).max() <= 1e-11 * np.abs(a[1]).max(), (a[1], b[1])


def test_poisoned_work_space_changes_nothing():
    N, nfile = 24, 20
    s0 = asd.random_spins(N, nfile, seed=9)
    target = np.array([0.5 + 0.1j, 0.3 - 0.1j])
    grads = []
    for poison in (False, True):
        with asd.Context(asd.Params.make(N, nfile, J1=1.0, alpha=0.1, dt=0.01),
                         modes=["fp64"]) as ctx:
            ctx.set_spins(s0, as_origin=True)
            ctx.loss_grad(6, 3, 4, target)
            if poison:
                ctx.debug_poison()
            grads.append(ctx.loss_grad(6, 3, 4, target))
    assert grads[0][0] == grads[1][0] and np.array_equal(grads[0][1], grads[1][1])
