"""The operators on the tables of a structured mesh and on a vertex mesh's faces
held once against the N x 6 array kernels, bit for bit.  The array side is a
vertex mesh (for a structured one, on the same lattice points with the
reference's formulas, which gives the same arrays) on which the arrays are
forced: they are built first, and a budget without room for anything else keeps
the faces away (checked: nothing but the stabilisation's scratch is allocated)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = [(1, 1, 1), (1, 4, 4), (2, 3, 5), (33, 7, 9), (5, 6, 130), (300, 1, 2), (1, 300, 3), (40, 31, 62), (17, 65, 33),
          (101, 79, 83), (88, 84, 96), (161, 95, 82)]
KINDS = ["tables", "faces", "faces_compat"]


def make(cfdb, ctx, shape, kind, arrays):
    h = 1.0 / max(shape)
    sp = (h, 1.25 * h, 0.8 * h)
    if kind == "tables" and not arrays:
        return cfdb.Mesh.structured(ctx, *shape, *sp)
    v = np.stack(np.meshgrid(*[np.arange(n + 1) * s for n, s in zip(shape, sp)], indexing="ij"), -1)
    if kind == "faces":  # component-sum areas make no closed cells of jittered vertices
        v += np.random.default_rng(9).uniform(-0.15, 0.15, v.shape) * h
    return cfdb.Mesh.from_vertices(ctx, *shape, *sp, v, compat_area=kind != "faces")


def field(n, dtype, seed):
    return torch.as_tensor(np.random.default_rng(seed).standard_normal(n), dtype=dtype, device=DEV)


def same(a, b):
    """Equal bits; any NaN for a NaN."""
    t = torch.int32 if a.dtype == torch.float32 else torch.int64
    na, nb = torch.isnan(a), torch.isnan(b)
    return torch.equal(na, nb) and torch.equal(torch.where(na, 0, a.view(t)), torch.where(nb, 0, b.view(t)))


class Sides:
    """One call on both geometries: its results on the form under test, then on the arrays."""

    def __init__(self, cfdb, shape, kind, dtype):
        self.cfdb = cfdb
        self.ctx = [cfdb.Context(0), cfdb.Context(0)]
        self.mesh = [make(cfdb, c, shape, kind, k == 1) for k, c in enumerate(self.ctx)]
        c, m = self.ctx[1], self.mesh[1]
        p = torch.zeros(m.n, dtype=dtype, device=DEV)
        c.boundary_copy(m, p, p)      # builds the arrays
        spare = c.allocated_bytes()
        c.set_alloc_budget(spare + 18 * p.element_size() * m.n)
        c.stab(m, p)                  # and their scratch
        assert c.allocated_bytes() == spare + 18 * p.element_size() * m.n, "the arrays do not serve"
        self.held = c.allocated_bytes()
        c.set_alloc_budget(self.held)

    def __call__(self, fn):
        out = [fn(c, m) for c, m in zip(self.ctx, self.mesh)]
        assert self.ctx[1].allocated_bytes() == self.held
        return out


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_operators(cfdb, shape, kind, dtype):
    both = Sides(cfdb, shape, kind, dtype)
    n = both.mesh[0].n
    tiny = 1e-36 if dtype == torch.float32 else 1e-300
    top = torch.finfo(dtype).max
    fields = [field(n, dtype, 1)]
    f = field(n, dtype, 2)            # sums around and below what the reciprocal divides, among ordinary ones
    f[: n // 3] *= tiny
    f[n // 2:: 3] *= tiny * 1e5
    fields.append(f)
    for value in (float("inf"), -float("inf"), float("nan"), top, -0.6 * top):
        f = field(n, dtype, 3)
        for i in (0, n // 2, n - 1):
            f[i] = value
        fields.append(f)
    for k, phi in enumerate(fields):
        for op in ("grad", "lapl", "stab"):
            for mask in (7, 1, 2, 4, 6, 0) if k < 2 else (7, 2, 0):
                got, ref = both(lambda c, m: getattr(c, op)(m, phi, mask=mask))
                assert same(got, ref), (op, mask, k)

        def heat(c, m):
            out = torch.empty_like(phi)
            c.heat_step(m, phi, out, 0.7, 1e-5, path=cfdb.PLAIN)
            return out
        assert same(*both(heat)), k


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_acoustic_step(cfdb, shape, dtype):
    both = Sides(cfdb, shape, "tables", dtype)
    n = both.mesh[0].n
    c_field = torch.exp(0.1 * field(n, dtype, 4))
    for value in (None, float("inf"), float("nan")):
        q = field(4 * n, dtype, 5)
        q[:n // 3] *= 1e-36 if dtype == torch.float32 else 1e-300
        if value is not None:
            for i in (0, 2 * n - 1, 2 * n + n // 2, 4 * n - 1):
                q[i] = value
        for cf, mode in ((None, 0), (None, 1), (c_field, 0), (c_field, 1)):
            def wave(c, m):
                out = torch.empty_like(q)
                c.wave_step(m, q, out, 1e-4, c=cf, c_const=0.9, speed_mode=mode, path=cfdb.PLAIN)
                return out
            assert same(*both(wave)), (value, mode)
