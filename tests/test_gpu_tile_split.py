"""Tiles whose particles are shared by several CTAs (few tiles, FP32) against
the same particles with every tile whole and against the oracle."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from oracle.oracle import Oracle
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


# one tile with far more particles than a CTA takes at once; a tile row with an
# empty end; counts around the 128 and NT (256 in 2D, 1024 in 3D) of the split
@pytest.mark.parametrize("order", [0, 1, 2, 3])
@pytest.mark.parametrize("n,cells,count", [
    ((16, 8, 1), 1, 20000), ((50, 20, 1), None, 3001), ((64, 64, 1), None, 65537), ((16, 16, 1), None, 511),
    ((16, 8, 8), None, 30001), ((17, 9, 24), None, 2049), ((24, 16, 8), 1, 5000)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 1, 1)])
def test_split_tiles(order, n, cells, count, periodic):
    dim = 2 if n[2] == 1 else 3
    bc = tuple((0, 0) if p else (2, 2) for p in periodic)
    g = GridSpec(dim=dim, n=n, order=order, real=torch.float32, periodic=periodic, prtl_bc=bc)
    EB = random_fields(g, 5, amp=0.2)
    o, ctx = Oracle(g), Context(g)
    o.fill_ghosts(EB, True, 0, 6)
    sp = []
    for k in range(2):
        m = max(count // (k + 1), 1)
        s = make_species(GridSpec(dim=dim, n=(m, 1, 1), order=2, real=g.real), 1, 0.4, 0.0, 7 + k,
                         charge=(-1.0) ** k, index=k + 1)
        gen = torch.Generator().manual_seed(count + k)
        for d in range(3):
            hi = g.n[d] if cells is None else min(cells + 1, g.n[d])
            s.i[d] = torch.randint(0, hi, (m,), generator=gen, dtype=torch.int32)
            s.dx[d] = torch.rand(m, generator=gen) if d < dim else torch.zeros(m)
        s.i_prev, s.dx_prev = [x.clone() for x in s.i], [x.clone() for x in s.dx]
        s.w = 0.5 + torch.rand(m, generator=gen)
        q = s.to("cuda")
        assert ctx.sort(q, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED) == abi.PIC_OK
        sp.append(q)
    cpu = [s.clone().to("cpu") for s in sp]
    Jo, Jg = empty_field(g, 3), empty_field(g, 3, "cuda")
    for s in cpu:
        o.push(s, EB, 0.45, 0.6, g.dx)
    o.deposit(cpu, Jo, 0.45, g.dx)
    ctx.push_deposit(sp, EB.cuda(), Jg, 0.45, 0.6, g.dx, flags=abi.PIC_PD_WRITE_PREV)
    torch.cuda.synchronize()
    for s, q in zip(cpu, sp):
        for a, b in zip(s.i[:dim] + s.dx[:dim] + s.u + [s.tag], q.i[:dim] + q.dx[:dim] + q.u + [q.tag]):
            assert torch.equal(a, b.cpu())
    o.sync_currents(Jo, empty_field(g, 3))
    o.fill_ghosts(Jo, False, 0, 3)
    ctx.sync_currents(Jg)
    scale = float(Jo.abs().max())
    # the bound of every deposit against the oracle: 4e-6; the oracle's float sum
    # of m particles in one cell adds sqrt(m) roundings of 2^-24
    tol = 4e-6 + 2.0 ** -24 * (count if cells else 64) ** 0.5
    assert float((Jo - Jg.cpu()).abs().max()) <= tol * scale
    assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
    ctx.close()
