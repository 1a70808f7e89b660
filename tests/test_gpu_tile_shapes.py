"""One fused FP32 step on meshes that between them take every tile shape of every
sweep, against the FP64 plain path (or, where the layer's operators give the same
bits, against those).  The rules that choose a tile are restated here, so that
the test itself says which shapes its meshes reach.  One step from O(1) fields
rounds to a few 1e-7; the bar is the fused paths' 1e-5."""
from __future__ import annotations

from math import ceil

import numpy as np
import pytest
import torch

DEV = "cuda:0"
SMS = 148

SHAPES = [(5, 19, 40), (16, 16, 256), (40, 16, 40), (40, 31, 80), (41, 40, 48), (42, 64, 32), (43, 33, 64), (44, 37, 100), (45, 24, 132), (46, 25, 120),
          (24, 29, 200), (30, 30, 128), (70, 20, 96), (37, 95, 44), (160, 48, 200), (36, 90, 224), (37, 200, 64)]


def cover(s, tz, ty):
    return ceil(s[2] / tz) * tz * ceil(s[1] / ty) * ty


def few(s):
    rows = ceil(s[1] / 8) * s[0]
    n32, n64 = ceil(s[2] / 32) * rows, ceil(s[2] / 64) * rows
    return 32 if n32 <= SMS else 64 if s[2] >= 64 and n64 <= SMS else 32 if n32 <= 2 * SMS else 0


def least(costs):
    return min(costs, key=lambda k: (costs[k], list(costs).index(k)))


def wave_tile(s, field):
    if few(s):
        return f"{few(s)}x8"
    narrow = field and ceil(s[2] / 128) * ceil(s[1] / 8) * s[0] > SMS
    return least({"128x8": (1.01 if narrow else 1.0) * cover(s, 128, 8), "64x8": (1.0 if narrow else 1.01) * cover(s, 64, 8),
                  "48x8": 1.15 * cover(s, 48, 8), "40x16": 1.15 * cover(s, 40, 16), "32x16": 1.08 * cover(s, 32, 16)})


def padded_tile(s, narrow):
    c = {"128x8": cover(s, 128, 8), "64x8": cover(s, 64, 8), "40x16": narrow * cover(s, 40, 16), "32x16": narrow * cover(s, 32, 16)}
    if s[2] < 128:
        del c["128x8"]
    return least(c)


def adjoint_tile(s):
    if few(s):
        return f"{few(s)}x8"
    c48, c64, c32 = 1.1 * cover(s, 48, 8), cover(s, 64, 8) / 0.94, cover(s, 32, 16)
    return "48x8" if c48 < c32 and c48 < c64 else "64x8" if c64 < c32 else "32x16"


def distorted_tile(s):
    if ceil(s[2] / 32) * ceil(s[1] / 8) * s[0] <= SMS:
        return "32x8 one"
    up = lambda t: ceil(s[2] / t) * t  # noqa: E731
    return least({"64x8": up(64), "96x4": 1.05 * up(96), "48x8": 1.13 * up(48), "32x8": 1.12 * up(32)})


def euler_tile(s):
    def time(tz, ty):
        tiles, slots = ceil(s[2] / tz) * ceil(s[1] / ty), 2 * SMS
        chunks = min(max(1, slots // tiles), s[0])
        planes, ctas = ceil(s[0] / chunks), tiles * chunks

        def one(n):
            if tz * ty == 256:
                return (4.8 if n > SMS else 4.2) + 0.9 * planes
            return 5.8 + 1.4 * planes if n > SMS else 4.6 + planes
        return ctas // slots * one(slots) + (one(ctas % slots) if ctas % slots else 0.0)
    a, b, c = time(64, 8), time(32, 16), time(32, 8)
    return "64x8" if a <= 1.03 * min(b, c) else "32x16" if b <= c else "32x8"


def test_every_shape_is_reached():
    wave = {"128x8", "64x8", "48x8", "40x16", "32x16", "32x8"}
    for field in (False, True):
        assert {wave_tile(s, field) for s in SHAPES} == wave
    for narrow in (1.07, 1.15):
        assert {padded_tile(s, narrow) for s in SHAPES} == {"128x8", "64x8", "40x16", "32x16"}
    assert {adjoint_tile(s) for s in SHAPES} == {"64x8", "48x8", "32x16", "32x8"}
    assert {distorted_tile(s) for s in SHAPES} == {"64x8", "96x4", "48x8", "32x8", "32x8 one"}
    assert {euler_tile(s) for s in SHAPES} == {"64x8", "32x16", "32x8"}


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


def field(n, rng):
    return torch.as_tensor(rng.standard_normal(n), dtype=torch.float64, device=DEV)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_fused_steps(cfdb, ctx, shape):
    n = shape[0] * shape[1] * shape[2]
    h = 1.0 / max(shape)
    rng = np.random.default_rng(n)
    q, lam = field(4 * n, rng), field(4 * n, rng)
    c = 1.0 + 0.5 * torch.tanh(field(n, rng))
    m = cfdb.Mesh.structured(ctx, *shape, h, h, h)
    dt = 0.1 * h
    for cc, mode in ((None, 0), (c, 0), (c, 1)):
        ref, got = torch.empty_like(q), torch.empty(4 * n, device=DEV)
        ctx.wave_step(m, q, ref, dt, c=cc, c_const=0.8, speed_mode=mode, path=cfdb.PLAIN)
        ctx.wave_step(m, q.float(), got, dt, c=None if cc is None else cc.float(), c_const=0.8, speed_mode=mode)
        assert rel(got, ref) <= 1e-5, (cc is None, mode)
    refs = torch.empty_like(q), torch.zeros_like(c)
    gots = torch.empty(4 * n, device=DEV), torch.zeros(n, device=DEV)
    ctx.wave_adjoint_step(m, q, lam, refs[0], c, refs[1], dt, path=cfdb.PLAIN)
    ctx.wave_adjoint_step(m, q.float(), lam.float(), gots[0], c.float(), gots[1], dt)
    assert rel(gots[0], refs[0]) <= 1e-5 and rel(gots[1], refs[1]) <= 1e-5

    v = np.stack(np.meshgrid(*[np.arange(k + 1) * h for k in shape], indexing="ij"), -1)
    v[1:-1, 1:-1, 1:-1] += rng.uniform(-0.2, 0.2, v[1:-1, 1:-1, 1:-1].shape) * h
    d = cfdb.Mesh.from_vertices(ctx, *shape, h, h, h, v)
    ref, got = torch.empty_like(q), torch.empty(4 * n, device=DEV)
    ctx.wave_step(d, q, ref, dt, path=cfdb.PLAIN)
    ctx.wave_step(d, q.float(), got, dt)
    assert rel(got, ref) <= 1e-5

    u = field(n, rng).float()
    unit = cfdb.Mesh.structured(ctx, *shape, 1.0, 1.0, 1.0)
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
    out = []
    for x, dtype, path in ((U, cfdb.F64, cfdb.PLAIN), (U.float(), cfdb.F32, cfdb.FUSED)):
        e = cfdb.Euler(ctx, m, dtype, path, 1.4, 0.4, 1.0, 10)
        y, z = torch.empty_like(x), x.clone()
        e.begin(z)
        e.step(z, y)
        e.step(y, z)
        out.append((y, z, e.totals()))
        e.close()
    assert rel(out[1][0], out[0][0]) <= 1e-5 and rel(out[1][1], out[0][1]) <= 1e-5
    assert np.allclose(out[1][2], out[0][2], rtol=1e-5, atol=0)
