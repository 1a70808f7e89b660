"""What the geometries behind the per-operator calls ask of device memory:
calls that went through with the N x 6 arrays alone go through whatever ran
on the mesh before, inside a recorded graph and under an allocation budget."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPE, H = (17, 9, 33), 1.0 / 32


def make(cfdb, ctx, uniform):
    if uniform:
        return cfdb.Mesh.structured(ctx, *SHAPE, H, H, H)
    v = np.stack(np.meshgrid(*[np.arange(n + 1) * H for n in SHAPE], indexing="ij"), -1)
    v += np.random.default_rng(9).uniform(-0.2, 0.2, v.shape) * H
    return cfdb.Mesh.from_vertices(ctx, *SHAPE, H, H, H, v)


def field(m, dtype, seed):
    return torch.as_tensor(np.random.default_rng(seed).standard_normal(m.n), dtype=dtype, device=DEV)


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_stab_after_a_heat_step_needs_no_memory(cfdb, uniform, dtype):
    ctx = cfdb.Context(0)
    m = make(cfdb, ctx, uniform)
    phi = field(m, dtype, 1)
    want = ctx.stab(make(cfdb, ctx, uniform), phi)
    ctx.heat_step(m, phi, torch.empty_like(phi), 0.01, 1e-5, path=cfdb.PLAIN)
    ctx.sync()
    ctx.set_alloc_budget(ctx.allocated_bytes())
    assert torch.equal(ctx.stab(m, phi), want)
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ctx.set_stream(side.cuda_stream)
        got = ctx.stab(m, phi)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    graph.replay()
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_arrays_built_after_a_build_that_ran_out_of_memory(cfdb, dtype):
    """A first build that finds no room for any one of its allocations leaves
    nothing behind that a later one would take for filled."""
    ctx = cfdb.Context(0)
    es = 4 if dtype == torch.float32 else 8
    want = None
    for short in (0, 1, 2):
        m = make(cfdb, ctx, False)
        q = torch.as_tensor(np.random.default_rng(2).standard_normal(4 * m.n), dtype=dtype, device=DEV)
        out = torch.empty_like(q)
        if short:
            arrays = 56 * m.n * es + (24 * m.n if short == 2 else 0)
            ctx.set_alloc_budget(ctx.allocated_bytes() + arrays + 64)
            with pytest.raises(cfdb.CfdbError) as e:
                ctx.wave_step(m, q, out, 1e-3, path=cfdb.PLAIN)
            assert e.value.code == cfdb.capi.ENOMEM
            ctx.set_alloc_budget(0)
        ctx.wave_step(m, q, out, 1e-3, path=cfdb.PLAIN)
        ctx.sync()
        m.close()
        want = out if want is None else want
        assert torch.equal(out, want)
    ctx.sync()
