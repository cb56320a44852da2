"""Tiles whose particles several CTAs share against the same tiles left to one CTA
(ENTITY_PIC_NO_SPLIT=1): J and every particle to the bit. Order 0 has no record
buffers, so its tiles are never shared: the two runs are one route."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2, 3])
# one tile of many particles; counts around the 128 and NT (256 in 2D, 1024 in 3D) of
# the split; tiles without particles; more tiles than CTAs (not shared)
@pytest.mark.parametrize("n,cells,count", [
    ((16, 8, 1), 1, 20000), ((50, 20, 1), None, 3001), ((64, 64, 1), None, 65537), ((16, 16, 1), None, 513),
    ((16, 8, 8), None, 30001), ((17, 9, 24), None, 2049), ((24, 16, 8), 1, 5000), ((40, 48, 33), None, 200003),
    ((512, 256, 1), None, 400000)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 1, 1)])
def test_split_and_whole_tiles_agree(order, n, cells, count, periodic, monkeypatch):
    dim = 2 if n[2] == 1 else 3
    bc = tuple((0, 0) if p else (2, 2) for p in periodic)
    g = GridSpec(dim=dim, n=n, order=order, real=torch.float32, periodic=periodic, prtl_bc=bc)
    EB = random_fields(g, 5, amp=0.2).cuda()
    ctx = Context(g)
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
    got = []
    for off in ("0", "1"):
        monkeypatch.setenv("ENTITY_PIC_NO_SPLIT", off)
        here, J = [s.clone() for s in sp], empty_field(g, 3, "cuda")
        for _ in range(2):
            ctx.push_deposit(here, EB, J, 0.45, 0.6, g.dx, flags=abi.PIC_PD_WRITE_PREV)
        torch.cuda.synchronize()
        got.append((J, here))
    (Ja, a), (Jb, b) = got
    assert float(Ja.abs().max()) > 0 and torch.equal(Ja, Jb)
    for x, y in zip(a, b):
        for p, q in zip(x.i[:dim] + x.dx[:dim] + x.u + x.i_prev[:dim] + x.dx_prev[:dim] + [x.tag],
                        y.i[:dim] + y.dx[:dim] + y.u + y.i_prev[:dim] + y.dx_prev[:dim] + [y.tag]):
            assert torch.equal(p, q)
    assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
    ctx.close()
