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


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("first", ["grad", "lapl", "stab", "heat", "total"])
def test_a_budget_for_the_arrays_serves_every_call(cfdb, uniform, dtype, first):
    """A budget that holds the N x 6 arrays and the stabilisation's scratch, but
    no second geometry beside them: whichever operator comes first, the calls
    that need the arrays still go through."""
    ctx = cfdb.Context(0)
    ref = make(cfdb, ctx, uniform)
    phi = field(ref, dtype, 1)
    lam = torch.as_tensor(np.random.default_rng(2).standard_normal(4 * ref.n), dtype=dtype, device=DEV)

    def call(m, name):
        if name == "total":
            return torch.tensor(ctx.total_fp64(m, phi))
        if name == "heat":
            out = torch.empty_like(phi)
            ctx.heat_step(m, phi, out, 0.01, 1e-5, path=cfdb.PLAIN)
            return out
        if name == "adjoint":
            out, gc = torch.empty_like(lam), torch.zeros_like(phi)
            ctx.wave_adjoint_step(m, lam, lam * 0.5, out, phi * phi + 1, gc, 1e-3, path=cfdb.PLAIN)
            return torch.cat([out, gc])
        return getattr(ctx, name)(m, phi)

    names = [first, "adjoint", "grad", "stab"]
    want = [call(ref, n) for n in names]
    ctx.sync()
    ref.close()
    m = make(cfdb, ctx, uniform)
    es = phi.element_size()
    verts = 0 if uniform else 24 * (SHAPE[0] + 1) * (SHAPE[1] + 1) * (SHAPE[2] + 1)
    # the arrays (56 values per cell), the ids, then the larger of the vertices' copy and the scratch
    ctx.set_alloc_budget(ctx.allocated_bytes() + (56 * es + 24) * m.n + max(verts, 18 * es * m.n) + 64)
    for n, w in zip(names, want):
        got = call(m, n)
        assert torch.allclose(got, w, rtol=1e-12, atol=0) if n == "total" else torch.equal(got, w), n
    ctx.sync()
