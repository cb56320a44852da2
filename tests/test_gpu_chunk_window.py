"""Push + deposit without a tile binning (2D, FP32): blocks of consecutive
particles deposit through a window where they lie together. Against the oracle,
for orders of the particles that the window holds, does not hold, or holds in
part, across periodic edges, on non-periodic axes, and at block remainders."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from oracle.oracle import Oracle
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


def _species(g, n, layout, seed):
    s = make_species(GridSpec(dim=2, n=(n, 1, 1), order=2, real=g.real), 1, 0.4, 0.0, seed)
    gen = torch.Generator().manual_seed(seed)
    r = [torch.randint(0, g.n[d], (n,), generator=gen, dtype=torch.int32) for d in range(2)]
    if layout == "ordered":
        key = torch.sort(r[0].long() * g.n[1] + r[1].long()).values
        r = [(key // g.n[1]).to(torch.int32), (key % g.n[1]).to(torch.int32)]
    elif layout == "edge":  # around a periodic corner, a few elsewhere
        far = torch.rand(n, generator=gen) < 0.02
        r = [torch.where(far, x, (x % 5 - 2) % g.n[d]).to(torch.int32) for d, x in enumerate(r)]
    for d in range(2):
        s.i[d], s.dx[d] = r[d], torch.rand(n, generator=gen)
    s.i[2], s.dx[2] = torch.zeros(n, dtype=torch.int32), torch.zeros(n)
    s.i_prev, s.dx_prev = [x.clone() for x in s.i], [x.clone() for x in s.dx]
    s.tag[torch.rand(n, generator=gen) < 0.05] = 0
    return s


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("layout", ["random", "ordered", "edge"])
@pytest.mark.parametrize("bc", ["periodic", "absorb", "reflect"])
def test_chunk_window(order, layout, bc):
    k = {"periodic": 0, "absorb": 1, "reflect": 2}[bc]
    g = GridSpec(dim=2, n=(61, 83, 1), order=order, real=torch.float32,
                 periodic=(1, int(k == 0), 1), prtl_bc=((0, 0), (k, k), (0, 0)))
    EB = random_fields(g, 3, amp=0.2)
    for n in (1, 257, 5063, 61 * 83 * 5 + 100):
        o, ctx = Oracle(g), Context(g)
        o.fill_ghosts(EB, True, 0, 6)
        s = _species(g, n, layout, 11 * n + order)
        s.tag[0] = 1
        q = s.clone().to("cuda")
        Jo, Jg = empty_field(g, 3), empty_field(g, 3, "cuda")
        o.push(s, EB, 0.45, 0.6, g.dx)
        o.deposit([s], Jo, 0.45, g.dx)
        ctx.push_deposit([q], EB.cuda(), Jg, 0.45, 0.6, g.dx, flags=abi.PIC_PD_WRITE_PREV)
        torch.cuda.synchronize()
        # an absorbed particle keeps its slot; its arrays are compared too
        for a, b in zip(s.i[:2] + s.dx[:2] + s.u + s.i_prev[:2] + s.dx_prev[:2] + [s.tag],
                        q.i[:2] + q.dx[:2] + q.u + q.i_prev[:2] + q.dx_prev[:2] + [q.tag]):
            assert torch.equal(a, b.cpu())
        o.sync_currents(Jo, empty_field(g, 3))
        o.fill_ghosts(Jo, False, 0, 3)
        ctx.sync_currents(Jg)
        scale = float(Jo.abs().max())
        # the bound of every deposit against the oracle (test_gpu_parity): 4e-6
        assert float((Jo - Jg.cpu()).abs().max()) <= 4e-6 * max(scale, 1e-30), n
        assert ctx.device_errors() == [0, 0, 0, 0]
        ctx.close()
