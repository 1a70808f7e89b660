"""The operators and plain steps on structured meshes without face arrays
against the face-array kernels: a vertex mesh on the same lattice points with
the reference's formulas has the same face arrays and takes the array
kernels, so both must give the same bits (sizes around one cell per
direction, ragged columns, several planes per thread; operands that are not
finite or overflow)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
SHAPES = [((1, 1, 1), (0.5, 0.3, 0.2)), ((1, 4, 4), (1.0, 1.0, 1.0)), ((2, 3, 5), (1 / 13, 0.3, 1 / 7)),
          ((33, 7, 9), (1 / 33, 1 / 33, 1 / 33)), ((5, 6, 130), (0.01, 0.02, 0.03)), ((101, 79, 83), (1 / 101, 1 / 101, 1 / 101)),
          ((88, 84, 96), (0.125, 0.25, 0.5)), ((161, 95, 82), (1.0, 1.0, 1.0))]


def pair(cfdb, ctx, shape, spacing):
    ax = [np.arange(n + 1) * h for n, h in zip(shape, spacing)]
    v = np.stack(np.meshgrid(*ax, indexing="ij"), -1)
    return (cfdb.Mesh.structured(ctx, *shape, *spacing),
            cfdb.Mesh.from_vertices(ctx, *shape, *spacing, v, compat_area=True))


def same_bits(a, b):
    t = torch.int32 if a.dtype == torch.float32 else torch.int64
    return torch.equal(a.view(t), b.view(t))


def field(n, dtype, seed, scale=1.0):
    return torch.as_tensor(scale * np.random.default_rng(seed).standard_normal(n), dtype=dtype, device=DEV)


@pytest.mark.parametrize("shape,spacing", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_operators_equal_the_face_arrays(cfdb, ctx, shape, spacing, dtype):
    m, a = pair(cfdb, ctx, shape, spacing)
    phi = field(m.n, dtype, 1)
    phi[: m.n // 3] *= 1e-36 if dtype == torch.float32 else 1e-300  # sums below the reciprocal's range
    for op in ("grad", "lapl", "stab"):
        for mask in (7, 1, 2, 4, 6, 0):
            got, ref = (getattr(ctx, op)(k, phi, mask=mask) for k in (m, a))
            assert same_bits(got, ref), (op, mask)
    out = [torch.empty_like(phi) for _ in range(2)]
    for k, o in zip((m, a), out):
        ctx.heat_step(k, phi, o, 0.7, 1e-5, path=cfdb.PLAIN)
    assert same_bits(*out)
    q = field(4 * m.n, dtype, 3)
    cf = torch.exp(field(m.n, dtype, 4, 0.1))
    out = [torch.empty_like(q) for _ in range(2)]
    for c, mode in ((None, 0), (None, 1), (cf, 0), (cf, 1)):
        for k, o in zip((m, a), out):
            ctx.wave_step(k, q, o, 1e-4, c=c, c_const=0.9, speed_mode=mode, path=cfdb.PLAIN)
        assert same_bits(*out), mode


@pytest.mark.parametrize("shape,spacing", [((9, 8, 11), (0.1, 0.1, 0.1)), ((101, 79, 83), (1 / 101, 1 / 101, 1 / 101))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_operators_on_values_that_are_not_finite(cfdb, ctx, shape, spacing, dtype):
    m, a = pair(cfdb, ctx, shape, spacing)
    top = torch.finfo(dtype).max
    for value in (float("inf"), float("nan"), -float("inf"), top, -0.6 * top):
        phi = field(m.n, dtype, 2)
        for i in (0, m.n // 2 + 3, m.n - 1):
            phi[i] = value
        for op in ("grad", "lapl", "stab"):
            for mask in (7, 2, 0):
                got, ref = (getattr(ctx, op)(k, phi, mask=mask) for k in (m, a))
                assert torch.equal(torch.isnan(got), torch.isnan(ref)), (op, mask, value)
                assert torch.equal(torch.nan_to_num(got, nan=0.0), torch.nan_to_num(ref, nan=0.0)), (op, mask, value)
        q = field(4 * m.n, dtype, 5)
        for i in (0, 2 * m.n - 1, 2 * m.n + m.n // 2, 4 * m.n - 40):
            q[i] = value
        out = [torch.empty_like(q) for _ in range(2)]
        for k, o in zip((m, a), out):
            ctx.wave_step(k, q, o, 1e-4, c_const=0.9, path=cfdb.PLAIN)
        assert torch.equal(torch.isnan(out[0]), torch.isnan(out[1])), value
        assert torch.equal(torch.nan_to_num(out[0], nan=0.0), torch.nan_to_num(out[1], nan=0.0)), value


@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 3, 5), (17, 9, 33), (40, 31, 62)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_faces_held_once_equal_the_face_arrays(cfdb, ctx, shape, dtype):
    """Vertex meshes with every face's geometry held once against the N x 6
    arrays: the same jittered mesh scaled by 2^-30 has volumes outside the
    range of the reciprocal division and keeps the arrays, and every result
    scales by an exact power of two."""
    rng = np.random.default_rng(9)
    h = 1.0 / 64
    ax = [np.arange(n + 1) * h for n in shape]
    v = np.stack(np.meshgrid(*ax, indexing="ij"), -1)
    v += rng.uniform(-0.2, 0.2, v.shape) * h
    s = 2.0 ** -30
    m = cfdb.Mesh.from_vertices(ctx, *shape, h, h, h, v)
    a = cfdb.Mesh.from_vertices(ctx, *shape, h * s, h * s, h * s, v * s)
    for bad in (None, float("inf"), float("nan")):
        phi = field(m.n, dtype, 6)
        if bad is not None:
            phi[m.n // 2] = bad
        for op, scale in (("grad", s), ("lapl", s * s), ("stab", s)):
            for mask in (7, 1, 6, 0):
                got = getattr(ctx, op)(m, phi, mask=mask)
                ref = getattr(ctx, op)(a, phi, mask=mask) * scale
                assert torch.equal(torch.isnan(got), torch.isnan(ref)), (op, mask, bad)
                assert torch.equal(torch.nan_to_num(got, nan=0.0), torch.nan_to_num(ref, nan=0.0)), (op, mask, bad)
    phi = field(m.n, dtype, 7)
    out = [torch.empty_like(phi) for _ in range(2)]
    ctx.heat_step(m, phi, out[0], 0.7, 1e-5, path=cfdb.PLAIN)
    ctx.heat_step(a, phi, out[1], 0.7, 1e-5 * s * s, path=cfdb.PLAIN)
    assert torch.equal(*out)
    assert ctx.total_fp64(m, phi) == pytest.approx(ctx.total_fp64(a, phi) / s ** 3, rel=1e-12)


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_arrays_serve_when_nothing_else_can_be_built(cfdb, uniform, dtype):
    """With the N x 6 arrays there and no memory left, or while a graph is being
    recorded, the operators take the arrays: the same bits as the tables'."""
    shape, h = (17, 9, 33), 1.0 / 32
    v = np.stack(np.meshgrid(*[np.arange(n + 1) * h for n in shape], indexing="ij"), -1)
    v += np.random.default_rng(9).uniform(-0.2, 0.2, v.shape) * h
    ctx = cfdb.Context(0)

    def mesh():
        return cfdb.Mesh.structured(ctx, *shape, h, h, h) if uniform else cfdb.Mesh.from_vertices(ctx, *shape, h, h, h, v)

    def results(m):
        return [ctx.grad(m, phi), ctx.lapl(m, phi)]

    phi = field(shape[0] * shape[1] * shape[2], dtype, 6)
    want = results(mesh())
    m = mesh()
    ctx.boundary_copy(m, phi, phi)  # builds the arrays
    torch.cuda.synchronize()
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        ctx.set_stream(side.cuda_stream)
        recorded = results(m)
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    graph.replay()
    assert all(same_bits(a, b) for a, b in zip(recorded, want))
    ctx.set_alloc_budget(ctx.allocated_bytes())
    assert all(same_bits(a, b) for a, b in zip(results(m), want))
    ctx.set_alloc_budget(0)
    assert all(same_bits(a, b) for a, b in zip(results(m), want))


@pytest.mark.parametrize("shape,spacing", SHAPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_euler_step_equals_the_face_arrays(cfdb, ctx, shape, spacing, dtype):
    """The plain Euler step, dt and totals included: random states, momenta of
    zero and far from the others' range, a cell that turns out not finite."""
    m, a = pair(cfdb, ctx, shape, spacing)
    n = m.n
    code = cfdb.F64 if dtype == torch.float64 else cfdb.F32
    rng = np.random.default_rng(12)
    q = np.stack([rng.uniform(0.5, 2.0, n), *rng.standard_normal((3, n)), rng.uniform(20.0, 30.0, n)])
    q[2, ::3] = 0.0
    q[3, ::5] *= 1e-25
    plain = torch.as_tensor(q.reshape(-1), dtype=dtype, device=DEV)
    for i, bad in ((None, 0.0), (0 * n + n // 2, float("nan")), (2 * n + n // 3, float("inf")),
                   (4 * n + n - 1, -float("inf")), (n // 2, -1.0)):
        U = plain.clone()
        if i is not None:
            U[i] = bad
        out = []
        for mesh in (m, a):
            e = cfdb.Euler(ctx, mesh, code, cfdb.PLAIN, 1.4, 0.4, 1e9, 100)
            x, y = U.clone(), torch.full_like(U, 7.0)
            e.begin(plain)  # a finite first dt
            e.step(x, y)
            if i is None:
                for _ in range(2):
                    x, y = y, x
                    e.step(x, y)
                out.append((y, e.status(), e.totals()))
            else:
                out.append((y, None, None))
        ctx.sync()
        (y0, s0, t0), (y1, s1, t1) = out
        assert torch.equal(torch.isnan(y0), torch.isnan(y1)), i
        assert torch.equal(torch.nan_to_num(y0, nan=0.0), torch.nan_to_num(y1, nan=0.0)), i
        if i is None:
            assert s0 == s1 and np.array_equal(t0, t1)
