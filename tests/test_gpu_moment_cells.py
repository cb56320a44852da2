"""Output moments of many particles (the shared-window kernel) cell by cell: every
node against a 64-bit sum, relative to the sum of its contributions' magnitudes,
where small coefficients have cells of their own beside large ones."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context

pytestmark = pytest.mark.gpu

# More particles than the direct kernel takes, with a remainder of the chunks of 4096.
COUNT = 80 * 4096 + 123
# Roundings of 2^-24: the coefficient 12, the constant shape 1, the products 3, a
# block's total 1, and one per block that adds to the node (up to 27 of the blocks
# of consecutive cells, all 81 where every particle is in one cell); the shape factors
# themselves are exact (offsets that are multiples of 1/32).
ROUND = 2.0 ** -24


def _particles(g, layout, seed):
    s = make_species(GridSpec(dim=g.dim, n=(COUNT, 1, 1), order=2, real=g.real), 1, 0.3, 0.0, seed,
                     device="cuda", with_prev=False)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda: torch.rand(COUNT, generator=gen, device="cuda")
    cells = g.ncells()
    c = (torch.arange(COUNT, device="cuda") * cells) // COUNT  # cell order
    if layout == "random":
        c = (rand() * cells).long()
    elif layout == "clump":  # a chunk's particles together but for some that drifted away
        c = torch.where(rand() < 0.02, (rand() * cells).long(), c)
    elif layout == "cell":
        c = torch.full_like(c, cells - 1)
    c = c.clamp(max=cells - 1)
    for d in range(3):
        n = g.n[d] if d < g.dim else 1
        s.i[d] = (c % n).to(torch.int32)
        c = c // n
        s.dx[d] = (torch.floor(rand() * 16) / 16 + 1 / 32) if d < g.dim else torch.zeros(COUNT, device="cuda")
    s.tag = torch.where(rand() < 0.05, 0, 1).to(torch.int16)
    return s, rand


def _reference(g, s, p):
    """The moment and the sum of magnitudes, in 64 bits, ghost-inclusive."""
    D, W = g.dim, (p.order + 1) // 2
    u = [x.double() for x in s.u]
    u0 = torch.sqrt(1 + sum(x * x for x in u))
    comp = lambda c: u[c - 1] if c > 0 else u0
    c = {abi.PIC_MOM_N: lambda: torch.ones_like(u0), abi.PIC_MOM_V: lambda: comp(p.c1) / u0,
         abi.PIC_MOM_T: lambda: comp(p.c1) * comp(p.c2) / u0}[p.id]()
    c = c * s.w.double() * p.inv_n0 / p.dx ** D * (s.tag == 1)
    S = []
    for d in range(D):
        row = []
        for q in range(2 * W + 1):
            x = (s.dx[d].double() - (q - W + 0.5)).abs()
            row.append(torch.full_like(x, 1 / (2 * W + 1)) if p.smoothing == abi.PIC_SMOOTH_CONST else
                       torch.ones_like(x) if p.order == 0 else
                       torch.where(x < 0.5, 0.75 - x * x, 0.5 * (1.5 - x).clamp_min(0) ** 2) if p.order == 2
                       else (1 - x).clamp_min(0))
        S.append(row)
    ext = tuple(reversed(g.ext))
    out = torch.zeros(2, ext[0] * ext[1] * ext[2], dtype=torch.float64, device="cuda")
    ng = [g.ng] * D + [0] * (3 - D)
    for t in range((2 * W + 1) ** D):
        k = [t // (2 * W + 1) ** d % (2 * W + 1) for d in range(D)] + [W] * (3 - D)
        v, at = c, 0
        for d in reversed(range(3)):
            at = at * g.ext[d] + s.i[d].long() + (k[d] - W if d < D else 0) + ng[d]
        for d in range(D):
            v = v * S[d][k[d]]
        out[0].index_add_(0, at, v)
        out[1].index_add_(0, at, v.abs())
    return out.reshape(2, *ext)


def _check(g, s, moments, roundings):
    ctx = Context(g)
    for mid, c1, c2, order, smoothing in moments:
        p = abi.PicMomentParams()
        p.id, p.c1, p.c2, p.order, p.smoothing = mid, c1, c2, order, smoothing
        p.use_weights, p.inv_n0, p.dx = 1, 0.5, 0.75
        buf = empty_field(g, 6, "cuda")
        ctx.output_moment([s], p, buf, 2)
        torch.cuda.synchronize()
        ref, mag = _reference(g, s, p)
        off = (buf[2].double() - ref).abs()
        assert float(mag.max()) > 0
        bad = off > roundings * ROUND * mag
        assert not bool(bad.any()), (mid, c1, order, int(bad.sum()), float((off / mag)[mag > 0].max()))
    assert ctx.device_errors() == [0, 0, 0, 0]
    ctx.close()


SPLINE, CONST = abi.PIC_SMOOTH_SPLINE, abi.PIC_SMOOTH_CONST
T, V, N = abi.PIC_MOM_T, abi.PIC_MOM_V, abi.PIC_MOM_N


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("ratio", [1e-1, 1e-2, 1e-3, 1e-4, 1e-7])
@pytest.mark.parametrize("where", ["halves", "mixed"])
def test_cold_cells_beside_hot_ones(dim, ratio, where):
    g = GridSpec(dim=dim, n=(16, 16, 256) if dim == 3 else (40, 1650, 1), order=2, real=torch.float32)
    s, _ = _particles(g, "cells", 7)
    cell = (s.i[2].long() * g.n[1] + s.i[1]) * g.n[0] + s.i[0]
    cold = s.i[0] >= g.n[0] // 2 if where == "halves" else (cell * 2654435761 >> 7) % 2 == 0
    for d in range(3):
        s.u[d] = torch.where(cold, s.u[d] * ratio, s.u[d])
    _check(g, s, [(T, 1, 1, 2, SPLINE), (T, 1, 2, 1, SPLINE), (V, 1, 0, 2, SPLINE), (T, 3, 3, 2, CONST)], 48)
    # the same by weights
    s.u = [u * 0 + 0.3 for u in s.u]
    s.w = torch.where(cold, s.w * ratio, s.w)
    _check(g, s, [(N, 0, 0, 2, SPLINE), (T, 0, 0, 1, CONST)], 48)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("layout", ["cells", "clump", "random", "cell"])
@pytest.mark.parametrize("weight", [1.0, 1e-30, 1e30])
def test_layouts(dim, layout, weight):
    g = GridSpec(dim=dim, n=(16, 16, 256) if dim == 3 else (40, 1650, 1), order=2, real=torch.float32)
    s, rand = _particles(g, layout, 9)
    s.w = (weight * (0.5 + rand().double())).float()
    # without a window an addition per particle: up to COUNT of them in one node; in
    # random order about 5 particles a cell, each touching 27 nodes, 200 at the most
    n = 20 + {"cells": 27, "clump": 27 + 40, "random": 200, "cell": 81}[layout]
    _check(g, s, [(N, 0, 0, 0, SPLINE), (N, 0, 0, 2, SPLINE), (T, 0, 1, 1, SPLINE), (V, 2, 0, 2, CONST)], n)


# the lines between the block sizes: three blocks of 2048 per SM of 152, 8 particles per cell
@pytest.mark.parametrize("dim,n,count", [
    (3, (40, 40, 73), 3 * 152 * 2048 - 1), (3, (40, 40, 73), 3 * 152 * 2048 + 2047), (3, (48, 48, 50), 8 * 48 * 48 * 50 - 1),
    (3, (48, 48, 50), 8 * 48 * 48 * 50 + 4097), (2, (320, 300, 1), 3 * 152 * 2048 + 1), (2, (70, 61, 1), 513), (3, (20, 18, 12), 33)])
@pytest.mark.parametrize("layout", ["cells", "clump"])
def test_block_sizes(dim, n, count, layout, monkeypatch):
    monkeypatch.setitem(globals(), "COUNT", count)
    g = GridSpec(dim=dim, n=n, order=2, real=torch.float32)
    s, rand = _particles(g, layout, 11)
    s.w = 0.5 + rand()
    # in these grids a chunk's cells may not fit a window: then every particle of the
    # 27 cells (9 to 30 each) adds by itself
    per = -(-count // g.ncells()) + 12
    _check(g, s, [(N, 0, 0, 2, SPLINE), (T, 1, 2, 2, CONST)], 20 + 27 * per)


@pytest.mark.parametrize("which", ["one", "all"])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf")])
def test_weights_that_are_not_finite(which, value):
    """They reach the nodes of their particles, and no others."""
    g = GridSpec(dim=3, n=(16, 16, 256), order=2, real=torch.float32)
    s, _ = _particles(g, "cells", 13)
    s.tag[:] = 1
    s.w[:] = 1.0
    at = slice(5000, 5001) if which == "one" else slice(0, 3 * 4096)
    if which == "all":
        s.w[at] = 0.0
    s.w[at] = value
    ctx = Context(g)
    p = abi.PicMomentParams()
    p.id, p.order, p.smoothing, p.use_weights, p.inv_n0, p.dx = N, 1, CONST, 1, 0.5, 0.75
    buf = empty_field(g, 6, "cuda")
    ctx.output_moment([s], p, buf, 0)
    torch.cuda.synchronize()
    hit = torch.zeros(buf[0].numel(), dtype=torch.bool, device="cuda")
    for k in range(27):
        d = [k % 3 - 1, k // 3 % 3 - 1, k // 9 - 1]
        flat = 0
        for a in reversed(range(3)):
            flat = flat * g.ext[a] + s.i[a][at].long() + d[a] + g.ng
        hit[flat] = True
    assert torch.equal(~torch.isfinite(buf[0]).reshape(-1), hit)
    assert float(buf[0][torch.isfinite(buf[0])].abs().max()) > 0
    ctx.close()

