"""Several heat steps per pass (cfdb_heat_run on fields too large for one
cluster) against the one-step sweep, bit for bit: every pass length, tiles with
and without walls on their sides, odd rows, single planes and columns, and the
buffers the result may and may not touch."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("shape", [(1, 128, 64), (2, 65, 128), (9, 127, 132), (33, 123, 248), (4, 1, 4096), (70, 129, 36),
                                   (160, 130, 100), (300, 33, 392)])
def test_passes_equal_single_steps(cfdb, ctx, shape):
    X, Y, Z = shape
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / Y, 1 / Z)
    T0 = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, m.n), dtype=torch.float32, device=DEV)
    T0[::7] = 0.0
    k, dt = 0.01, 0.1 * min(1 / X, 1 / Y, 1 / Z) ** 2 / 0.01
    p, q = T0.clone(), torch.empty_like(T0)
    for steps in range(1, 12):
        ctx.heat_step(m, p, q, k, dt)
        p, q = q, p
        for graph in (True, False):
            a, b = T0.clone(), torch.full_like(T0, float("nan"))
            final = ctx.heat_run(m, a, b, k, dt, steps, use_graph=graph)
            assert (final is b) == bool(steps & 1)
            assert torch.equal(final, p), steps
    ctx.sync()


def test_passes_without_a_workspace(cfdb):
    """A field small enough to leave the other buffer alone takes both buffers
    when the workspace for that cannot be had."""
    ctx = cfdb.Context(0)
    m = cfdb.Mesh.structured(ctx, 96, 80, 100, 0.01, 0.01, 0.01)
    T0 = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, m.n), dtype=torch.float32, device=DEV)
    for steps in (7, 8):
        a, b = T0.clone(), torch.empty_like(T0)
        want = ctx.heat_run(m, a, b, 0.01, 1e-4, steps).clone()
        ctx.set_alloc_budget(ctx.allocated_bytes() + m.n)
        a = T0.clone()
        assert torch.equal(ctx.heat_run(m, a, b, 0.01, 1e-4, steps), want)
        ctx.set_alloc_budget(0)
    ctx.sync()


@pytest.mark.parametrize("k", [0.01, -0.01])
@pytest.mark.parametrize("value", [float("inf"), -float("inf"), float("nan"), 3e38])
def test_passes_on_values_that_are_not_finite(cfdb, ctx, k, value):
    """Infinities on and beside every wall, with a conductivity of either sign
    (a negative one adds infinities of one sign, so a wall's inf - inf is what
    makes the cell NaN): the one-step sweep's results."""
    X, Y, Z = 40, 130, 68
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / Y, 1 / Z)
    T0 = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, (X, Y, Z)), dtype=torch.float32, device=DEV)
    for i in ((0, 5, 5), (0, 0, 0), (X - 1, 60, 30), (20, 0, 7), (20, Y - 1, 40), (9, 77, 0), (30, 99, Z - 1), (11, 40, 33)):
        T0[i] = value
    T0 = T0.reshape(-1).contiguous()
    dt = 0.1 * min(1 / X, 1 / Y, 1 / Z) ** 2 / 0.01
    p, q = T0.clone(), torch.empty_like(T0)
    for steps in range(1, 6):
        ctx.heat_step(m, p, q, k, dt)
        p, q = q, p
        a, b = T0.clone(), torch.empty_like(T0)
        got = ctx.heat_run(m, a, b, k, dt, steps)
        assert torch.equal(torch.isnan(got), torch.isnan(p)), steps
        assert torch.equal(torch.nan_to_num(got, nan=0.0), torch.nan_to_num(p, nan=0.0)), steps
    ctx.sync()


def test_short_runs_of_long_meshes_pay_no_search(cfdb, ctx):
    """The host's share of a call on a long thin field (the search for a plan
    had looked at 74 thousand of them, 0.5 ms, even for a single step)."""
    import time
    X, Y, Z = 8192, 16, 16
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / X, 1 / X)
    a = torch.rand(m.n, device=DEV)
    b = torch.empty_like(a)
    for steps in (1, 2, 5):
        ctx.heat_run(m, a, b, 0.01, 1e-8, steps)
        took = []
        for _ in range(9):
            ctx.sync()
            t = time.perf_counter()
            ctx.heat_run(m, a, b, 0.01, 1e-8, steps)
            took.append(time.perf_counter() - t)
        assert sorted(took)[4] < 200e-6, (steps, took)
    ctx.sync()


def launches_of(ctx, fn):
    before = ctx.launch_count()
    fn()
    return ctx.launch_count() - before


@pytest.mark.parametrize("shape,steps", [((96, 24, 24), 40), ((1000, 4, 4), 5), ((2000, 8, 8), 9), ((70, 8, 8), 50),
                                         ((65, 20, 20), 7), ((512, 16, 16), 30), ((257, 7, 12), 33), ((81, 9, 4), 20),
                                         ((1000, 1, 64), 6), ((160, 160, 4), 12), ((2048, 8, 16), 11)])
def test_long_thin_fields_run_in_one_launch(cfdb, ctx, shape, steps):
    """Fields of many small planes stay in one cluster's shared memory for the
    whole run: the one-step sweep's bits from a single launch, the other buffer
    left alone."""
    X, Y, Z = shape
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / Y, 1 / Z)
    T0 = torch.as_tensor(np.random.default_rng(3).uniform(-1, 1, m.n), dtype=torch.float32, device=DEV)
    k, dt = 0.01, 0.1 * min(1 / X, 1 / Y, 1 / Z) ** 2 / 0.01
    p, q = T0.clone(), torch.empty_like(T0)
    for s in range(steps):
        ctx.heat_step(m, p, q, k, dt)
        p, q = q, p
    a, b = T0.clone(), torch.full_like(T0, float("nan"))
    out = []
    assert launches_of(ctx, lambda: out.append(ctx.heat_run(m, a, b, k, dt, steps))) == 1
    assert torch.equal(out[0], p)
    assert torch.equal(a, T0) if steps & 1 else torch.isnan(b).all()
    ctx.sync()


@pytest.mark.parametrize("shape,steps,launches", [
    ((64, 64, 64), 37, 1), ((40, 36, 32), 12, 1), ((17, 24, 20), 9, 1), ((8, 8, 8), 1, 1), ((16, 64, 64), 6, 1),
    # beyond one cluster: as many passes of two or three steps as keep the parity
    ((128, 64, 64), 23, 9), ((40, 96, 64), 14, 6), ((128, 64, 64), 1, 1), ((128, 64, 64), 2, 2), ((40, 96, 64), 3, 1),
    ((128, 128, 128), 4, 2)])
def test_which_form_ran(cfdb, ctx, shape, steps, launches):
    """The number of launches tells a run on one cluster from passes and from
    single steps."""
    X, Y, Z = shape
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / Y, 1 / Z)
    a = torch.rand(m.n, device=DEV)
    b = torch.empty_like(a)
    for graph in (False, True):
        assert launches_of(ctx, lambda: ctx.heat_run(m, a, b, 0.01, 1e-7, steps, use_graph=graph)) == launches
    ctx.sync()


@pytest.mark.parametrize("shape", [(96, 96, 96), (100, 100, 100), (140, 128, 32), (200, 128, 128)])
def test_recorded_passes_allocate_nothing(cfdb, ctx, shape):
    """A run recorded into the caller's graph is kernels only, so that the graph
    can be instantiated and embedded as one of single steps can."""
    from cuda.bindings import runtime as rt
    X, Y, Z = shape
    m = cfdb.Mesh.structured(ctx, X, Y, Z, 1 / X, 1 / Y, 1 / Z)
    T0 = torch.rand(m.n, device=DEV)
    a, b = T0.clone(), torch.empty_like(T0)
    want = ctx.heat_run(m, a, b, 0.01, 1e-7, 7, use_graph=False).clone()
    a.copy_(T0)
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=side):
        ctx.set_stream(side.cuda_stream)
        got = ctx.heat_run(m, a, b, 0.01, 1e-7, 7, use_graph=False)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    handle = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, count = rt.cudaGraphGetNodes(handle)
    err, nodes, count = rt.cudaGraphGetNodes(handle, count)
    kinds = {rt.cudaGraphNodeGetType(n)[1] for n in nodes[:count]}
    assert kinds == {rt.cudaGraphNodeType.cudaGraphNodeTypeKernel}
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
