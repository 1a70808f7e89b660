"""One fused FP32 step on meshes that take each tile shape of the sweeps
(widths 32, 40, 48, 64, 96, 128 by row length, ragged in both directions)
against the FP64 plain path.  One step from O(1) fields rounds to a few 1e-7;
the bar is the fused paths' 1e-5."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("nz", [16, 32, 40, 48, 80, 96, 100, 132, 160, 200])
def test_fused_steps_on_every_tile(cfdb, ctx, nz):
    nx, ny = 5, 19
    n = nx * ny * nz
    h = 1.0 / nz
    rng = np.random.default_rng(nz)
    t64 = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    q, lam = t64(rng.standard_normal(4 * n)), t64(rng.standard_normal(4 * n))
    c = t64(rng.uniform(0.5, 1.5, n))
    m = cfdb.Mesh.structured(ctx, nx, ny, nz, h, h, h)
    dt = 0.1 * h
    for cc, mode in ((None, 0), (c, 0), (c, 1)):
        ref, got = torch.empty_like(q), torch.empty(4 * n, device=DEV)
        ctx.wave_step(m, q, ref, dt, c=cc, c_const=0.8, speed_mode=mode, path=cfdb.PLAIN)
        ctx.wave_step(m, q.float(), got, dt, c=None if cc is None else cc.float(), c_const=0.8, speed_mode=mode)
        assert rel(got, ref) <= 1e-5
    refs = torch.empty_like(q), torch.zeros_like(c)
    gots = torch.empty(4 * n, device=DEV), torch.zeros(n, device=DEV)
    ctx.wave_adjoint_step(m, q, lam, refs[0], c, refs[1], dt, path=cfdb.PLAIN)
    ctx.wave_adjoint_step(m, q.float(), lam.float(), gots[0], c.float(), gots[1], dt)
    assert rel(gots[0], refs[0]) <= 1e-5 and rel(gots[1], refs[1]) <= 1e-5

    ax = [np.arange(k + 1) * h for k in (nx, ny, nz)]
    v = np.stack(np.meshgrid(*ax, indexing="ij"), -1)
    v[1:-1, 1:-1, 1:-1] += rng.uniform(-0.2, 0.2, v[1:-1, 1:-1, 1:-1].shape) * h
    d = cfdb.Mesh.from_vertices(ctx, nx, ny, nz, h, h, h, v)
    ref, got = torch.empty_like(q), torch.empty(4 * n, device=DEV)
    ctx.wave_step(d, q, ref, dt, path=cfdb.PLAIN)
    ctx.wave_step(d, q.float(), got, dt)
    assert rel(got, ref) <= 1e-5

    u = t64(rng.standard_normal(n)).float()
    unit = cfdb.Mesh.structured(ctx, nx, ny, nz, 1.0, 1.0, 1.0)
    out, fixed = torch.empty(n, device=DEV), torch.empty(n, device=DEV)
    ctx.d2t_step(unit, u, u * 0.5, out, 0.7, [1, 2], 0.3)
    rhs = ctx.scalar(cfdb.capi.OP_MUL, ctx.binary(cfdb.capi.OP_ADD, ctx.lapl(unit, u, mask=1), ctx.lapl(unit, u, mask=2)), 0.7)
    assert torch.equal(out, ctx.d2t(rhs, u, u * 0.5, 0.3, 1))
    ctx.heat_step_fixed(unit, u, fixed, 0.1, 0.3, u * 2)
    ctx.heat_step(unit, u, out, 0.1, 0.3)
    ctx.boundary_set(unit, out, u * 2)
    assert torch.equal(fixed, out)

    U = torch.empty(5, n, dtype=torch.float64, device=DEV)
    U[0], U[1:4], U[4] = 1.0, 0.1 * q.reshape(4, n)[:3], 2.5
    U = U.reshape(-1)
    ref, got = torch.empty_like(U), torch.empty(5 * n, device=DEV)
    for x, o, dtype, path in ((U, ref, cfdb.F64, cfdb.PLAIN), (U.float(), got, cfdb.F32, cfdb.FUSED)):
        e = cfdb.Euler(ctx, m, dtype, path, 1.4, 0.4, 1.0, 10)
        e.begin(x)
        e.step(x, o)
        ctx.sync()
        e.close()
    assert rel(got, ref) <= 1e-5
