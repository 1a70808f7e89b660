"""The one-launch reductions (CFL step, conserved total) against torch in FP64:
one cell, remainders of the four-value loads, more CTAs than the fold has
threads; fields on and off 16-byte boundaries (the vector and the scalar form);
the cell that decides at the ends and in the remainder; large and small meshes
by turns on one context, whose scratch and ticket they share."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIZES = [(1, 1, 1), (1, 1, 3), (5, 1, 1), (7, 11, 13), (64, 64, 64), (97, 89, 83), (1, 1, 2), (131, 101, 67), (3, 3, 3)]


def field(n, dtype, rng, lo, hi, off):
    """n values that start `off` elements behind a 16-byte boundary."""
    t = torch.empty(n + 8, dtype=dtype, device=DEV)[off: off + n]
    t.copy_(torch.as_tensor(rng.uniform(lo, hi, n), dtype=dtype))
    return t


@pytest.mark.parametrize("off", [0, 1, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_cfl_step(cfdb, ctx, dtype, off):
    # a handful of roundings: the sound speed, |u|, their sum, a quotient, two products
    tol = 16 * torch.finfo(dtype).eps
    rng = np.random.default_rng(4)
    for shape in SIZES:
        n = shape[0] * shape[1] * shape[2]
        m = cfdb.Mesh.structured(ctx, *shape, 0.01, 0.02, 0.03)
        p, rho = field(n, dtype, rng, 0.5, 1.0, off), field(n, dtype, rng, 0.5, 1.0, off)
        vel = [field(n, dtype, rng, -0.3, 0.3, off) for _ in range(3)]
        for at in sorted({0, n - 1, n // 2, n // 4 * 4 % n, max(0, n - 2)}):
            keep = vel[0][at].clone()
            vel[0][at] = 7.0 + at % 5
            for use in (vel, vel[:1]):
                d = [t.double() for t in (p, rho, *use)]
                s = torch.sqrt(1.4 * d[0] / d[1]) + torch.sqrt(sum(x * x for x in d[2:]))
                want = 0.4 * 0.01 / float(s.max())
                got = ctx.cfl_dt(m, 0.4, 1.4, p, rho, *use)
                assert got == pytest.approx(want, rel=tol), (shape, at)
            vel[0][at] = keep


@pytest.mark.parametrize("vertices", [False, True])
@pytest.mark.parametrize("off", [0, 1, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_total(cfdb, ctx, dtype, off, vertices):
    rng = np.random.default_rng(5)
    for shape in SIZES:
        n = shape[0] * shape[1] * shape[2]
        h = 0.01
        if vertices:
            v = np.stack(np.meshgrid(*[np.arange(k + 1) * h for k in shape], indexing="ij"), -1)
            m = cfdb.Mesh.from_vertices(ctx, *shape, h, h, h, v + rng.uniform(-0.2, 0.2, v.shape) * h)
            vol = torch.as_tensor(m.geometry(cfdb.capi.GEOM_VOLUME), device=DEV).to(dtype).double()
        else:
            m = cfdb.Mesh.structured(ctx, *shape, h, 0.02, 0.03)
            vol = torch.full((n,), h * 0.02 * 0.03, dtype=torch.float64, device=DEV)
        f = field(n, dtype, rng, -1.0, 1.0, off)
        for at in sorted({0, n - 1, n // 4 * 4 % n}):
            f[at] = 1e6          # a partial sum that the rest has to survive
            x = f.double() * vol
            # one rounding per product, the sum compensated; torch's own sum is pairwise
            assert abs(ctx.total_fp64(m, f) - float(x.sum())) <= 32 * 2.0 ** -53 * float(x.abs().sum()), (shape, at)
            f[at] = 0.5
        m.close()
