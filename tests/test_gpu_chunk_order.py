"""Which 2D kernel takes an unbinned species is found out on the device: the
same particles in cell order (windows) and in random order (by particle), and
in an order between, give the same J and the same particles to the bit."""
import pytest
import torch

from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


# 8 and 12 per cell and 2^19 particles are the lines of the rule; a remainder of the
# chunks of 512; dead particles and particles outside the grid among them
@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("n,ppc,dead", [((512, 256, 1), 8, 0.0), ((256, 256, 1), 8, 0.0), ((255, 257, 1), 8, 0.0), ((300, 293, 1), 12, 0.2), ((256, 256, 1), 15, 0.0),
                                        ((97, 676, 1), 16, 0.01)])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (0, 1, 1)])
def test_layout_leaves_results_unchanged(order, n, ppc, dead, periodic):
    bc = tuple((0, 0) if p else (2, 2) for p in periodic)
    g = GridSpec(dim=2, n=n, order=order, real=torch.float32, periodic=periodic, prtl_bc=bc)
    EB = random_fields(g, 5, amp=0.2).cuda()
    base = make_species(g, ppc, 0.5, 0.2, 7, device="cuda", shuffle=False)
    gen = torch.Generator(device="cuda").manual_seed(3)
    N = base.npart
    base.w = 0.5 + torch.rand(N, generator=gen, device="cuda")
    r = torch.rand(N, generator=gen, device="cuda")
    base.tag[r < dead] = 0
    base.i[0][(r >= dead) & (r < dead * 1.01)] = n[0] + 5
    orders = {"cells": torch.arange(N, device="cuda"),
              "random": torch.randperm(N, generator=gen, device="cuda"),
              # cell order, a tenth of the particles exchanged with others
              "mixed": torch.where(r < 0.1, torch.arange(N, device="cuda").flip(0), torch.arange(N, device="cuda"))}
    sym = r < 0.1
    orders["mixed"] = torch.where(sym & sym.flip(0), orders["mixed"], orders["cells"])
    got = {}
    for name, perm in orders.items():
        ctx = Context(g)
        s = base.clone()
        for k in range(2):
            s.i[k], s.dx[k] = s.i[k][perm].contiguous(), s.dx[k][perm].contiguous()
        s.u = [x[perm].contiguous() for x in s.u]
        s.w, s.tag = s.w[perm].contiguous(), s.tag[perm].contiguous()
        J = empty_field(g, 3, "cuda")
        ctx.push_deposit([s], EB, J, 0.45, 0.6, g.dx)
        torch.cuda.synchronize()
        inv = torch.argsort(perm)
        got[name] = (J, [x[inv] for x in s.i[:2] + s.dx[:2] + s.u + [s.tag]], ctx.device_errors())
        ctx.close()
    assert float(got["cells"][0].abs().max()) > 0
    for name in ("random", "mixed"):
        assert torch.equal(got[name][0], got["cells"][0]), name
        assert all(torch.equal(a, b) for a, b in zip(got[name][1], got["cells"][1])), name
        assert got[name][2] == got["cells"][2]
