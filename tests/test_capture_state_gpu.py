"""Calls captured into a CUDA graph and replayed between uncaptured calls, on
lattices whose steps run as the one-launch step, which writes the new spins to a
second buffer."""
from __future__ import annotations

import numpy as np
import pytest

import asd_b200 as asd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KW = dict(J1=-1.0, alpha=0.1, dt=0.01)


def make(N, nfile, kernel, stream):
    ctx = asd.Context(asd.Params.make(N, nfile, **KW), modes=["fp64"])
    ctx.set_stream(stream.cuda_stream)
    ctx.set_llg_kernel(kernel)
    ctx.set_spins(asd.random_spins(N, nfile, seed=N), as_origin=True)
    return ctx


@pytest.mark.parametrize("N,nfile,kernel", [(12, 3, "fused"), (33, 20, "fused"), (128, 256, "auto")])
def test_replayed_grid_leaves_the_spins(N, nfile, kernel):
    """The q grid's work space is none of the two buffers that a step alternates
    between: a replay after an odd number of steps leaves the spins as they are."""
    stream = torch.cuda.Stream()
    grid = torch.zeros(2 * N * N, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with make(N, nfile, kernel, stream) as ctx, make(N, nfile, kernel, stream) as other:
        ctx.step(1)
        assert asd.load().asd_ctx_last_launches(ctx.handle) == 1
        other.step(1)
        ctx.sqt_grid("fp64")  # takes its work space
        ctx.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.sqt_grid_async("fp64", grid.data_ptr())
        for _ in range(2):
            for c in (ctx, other):
                c.step(1)
            ctx.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            assert np.array_equal(ctx.get_spins(), other.get_spins())
        del graph


@pytest.mark.parametrize("N,nfile", [(12, 3), (20, 40), (51, 17)])
def test_replayed_origin_is_the_one_sqt_uses(N, nfile):
    """A captured set_spins_device(as_origin) gives its replays' origins to the
    uncaptured S(q,t) and loss that follow them."""
    stream = torch.cuda.Stream()
    first, origin, other_spins = (asd.random_spins(N, nfile, seed=k) for k in (1, 2, 3))
    buf = torch.from_numpy(first.reshape(-1)).cuda()
    target = np.array([0.2 + 0.1j, 0.1 - 0.1j])
    torch.cuda.synchronize()
    with make(N, nfile, "auto", stream) as ctx, make(N, nfile, "auto", stream) as plain:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.set_spins_device(buf.data_ptr(), as_origin=True)
        for values in (first, origin):
            buf.copy_(torch.from_numpy(values.reshape(-1)))
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                graph.replay()
            plain.set_spins(values, as_origin=True)
            for c in (ctx, plain):
                c.set_spins(other_spins, as_origin=False)
                c.step(2)
            assert ctx.sqt("fp64") == plain.sqt("fp64")
            a, b = ctx.loss_grad(4, 2, 2, target), plain.loss_grad(4, 2, 2, target)
            assert a[0] == b[0] and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
        del graph


@pytest.mark.parametrize("N,nfile", [(12, 3), (20, 40)])
def test_backward_keeps_the_origin_of_its_forward(N, nfile):
    """A replay of {new origin, S(q,t)} between the loss's two passes does not
    reach the gradient, which belongs to the forward pass's origin."""
    stream = torch.cuda.Stream()
    first, second = (asd.random_spins(N, nfile, seed=k) for k in (1, 2))
    buf = torch.from_numpy(first.reshape(-1)).cuda()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    target = np.array([0.2 + 0.1j, 0.1 - 0.1j])
    torch.cuda.synchronize()
    with make(N, nfile, "auto", stream) as ctx, make(N, nfile, "auto", stream) as plain:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.set_spins_device(buf.data_ptr(), as_origin=True)
            ctx.sqt_async("fp64", out.data_ptr())
        for c in (ctx, plain):
            c.set_spins(first, as_origin=True)
            c.loss_forward(4, 2, 2, target)
        buf.copy_(torch.from_numpy(second.reshape(-1)))
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            graph.replay()
        a, b = ctx.loss_backward(target), plain.loss_backward(target)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
        del graph


@pytest.mark.parametrize("N,nfile,kernel", [(12, 3, "fused"), (33, 20, "fused"), (96, 300, "auto"),
                                            (20, 24, "auto"), (20, 24, "stages")])
@pytest.mark.parametrize("nsteps", [1, 2, 3])
def test_replays_and_calls_go_on_from_one_another(N, nfile, kernel, nsteps):
    """Replayed steps start from the spins that the last replay or uncaptured call
    left, S(q,t) and the q grid see them, and an uncaptured call sees the replay's."""
    stream = torch.cuda.Stream()
    sq = torch.zeros(2, dtype=torch.float64, device="cuda")
    grid = torch.zeros(2 * N * N, dtype=torch.float64, device="cuda")
    spins = torch.zeros(nfile * N * N * 3, dtype=torch.float64, device="cuda")
    host = torch.zeros(nfile * N * N * 3, dtype=torch.float64).pin_memory()
    torch.cuda.synchronize()
    with make(N, nfile, kernel, stream) as ctx, make(N, nfile, kernel, stream) as plain:
        if N == 96:  # the default takes the one-launch step here
            ctx.step(2), plain.step(2)
            assert asd.load().asd_ctx_last_launches(ctx.handle) == 2
        for c in (ctx, plain):
            c.step(1)
            c.sqt("fp64"), c.sqt_grid("fp64")  # take their work space
            c.step_host(host.data_ptr(), host.data_ptr(), "fp64")
            c.set_spins(asd.random_spins(N, nfile, seed=7), as_origin=True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            ctx.step(nsteps)
            ctx.sqt_async("fp64", sq.data_ptr())
            ctx.sqt_grid_async("fp64", grid.data_ptr())
            ctx.get_spins_device(spins.data_ptr())

        def replay():
            with torch.cuda.stream(stream):
                graph.replay()
            stream.synchronize()
            plain.step(nsteps)
            assert complex(*sq.tolist()) == plain.sqt("fp64")
            assert np.array_equal(grid.cpu().numpy().view(complex).reshape(N, N),
                                  plain.sqt_grid("fp64"))
            y = plain.get_spins()
            assert np.array_equal(spins.cpu().numpy(), y.reshape(-1))
            assert np.array_equal(ctx.get_spins(), y)

        for _ in range(3):
            replay()
        for between in (lambda c: c.step(1), lambda c: c.step(2),
                        lambda c: c.step_host(host.data_ptr(), host.data_ptr(), "fp64")):
            for c in (ctx, plain):
                host.copy_(torch.from_numpy(plain.get_spins().reshape(-1)))
                between(c)
                torch.cuda.synchronize()
            replay()
            replay()
        del graph


@pytest.mark.parametrize("call", ["sqt", "grid", "split_grid"])
def test_first_call_captured_and_never_replayed(call):
    """In relaxed mode a first call may be captured: it takes its work space there.
    Uncaptured calls that follow find the fixed contents of that work space (a zero
    count, the twiddles) although the graph has not run."""
    N, nfile = 51, 9
    mode = "fp16x3" if call == "split_grid" else "fp64"
    stream = torch.cuda.Stream()
    out = torch.zeros(2 * N * N, dtype=torch.float64, device="cuda")
    params = asd.Params.make(N, nfile, **KW)
    with asd.Context(params, modes=[mode]) as ctx, asd.Context(params, modes=[mode]) as plain:
        for c in (ctx, plain):
            c.set_stream(stream.cuda_stream)
            c.set_spins(asd.random_spins(N, nfile, seed=1), as_origin=True)
        held = [torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda")
                for n in [4 << 10] * 64 + [1 << 20] * 32]
        torch.cuda.synchronize()
        del held
        torch.cuda.empty_cache()  # what the first call is given is not zero by chance
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="relaxed"):
            if call == "sqt":
                ctx.sqt_async(mode, out.data_ptr())
            else:
                ctx.sqt_grid_async(mode, out.data_ptr())
        for c in (ctx, plain):
            c.set_spins(asd.random_spins(N, nfile, seed=2), as_origin=True)
        if call == "sqt":
            assert ctx.sqt(mode) == plain.sqt(mode)
        else:
            assert np.array_equal(ctx.sqt_grid(mode), plain.sqt_grid(mode))
        ctx.check_device_status()
        del graph
