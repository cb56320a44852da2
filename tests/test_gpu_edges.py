"""Field kernels that visit only the cells near periodic edges, the 3D filter's
march along x3 and the conversion of the exact sums, at the smallest grids,
tile remainders and mixed periodic axes, against the oracle bit for bit."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from oracle.oracle import Oracle
from tests.helpers import random_currents, random_fields

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 1), (33, 7, 1), (61, 83, 1), (4, 4, 4), (5, 9, 4), (33, 9, 17), (70, 8, 35)]


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
@pytest.mark.parametrize("periodic", [(1, 1, 1), (1, 0, 1), (0, 1, 0), (0, 0, 1)])
@pytest.mark.parametrize("n", SHAPES)
def test_edges_and_filter(n, periodic, real):
    dim = 2 if n[2] == 1 else 3
    g = GridSpec(dim=dim, n=n, order=2, real=real, periodic=periodic,
                 prtl_bc=tuple((0, 0) if p else (1, 1) for p in periodic))
    o, ctx = Oracle(g), Context(g)
    Jo, buff = random_currents(g, 7), empty_field(g, 3)
    Jg, bg = Jo.cuda(), empty_field(g, 3, "cuda")
    o.sync_currents(Jo, buff)
    o.fill_ghosts(Jo, False, 0, 3)
    ctx.sync_currents(Jg, bg)
    torch.cuda.synchronize()
    assert torch.equal(Jo, Jg.cpu())
    for _ in range(3):
        o.filter_pass(Jo, buff)
        o.fill_ghosts(Jo, False, 0, 3)
    ctx.filter_currents(Jg, bg, 3)
    torch.cuda.synchronize()
    assert torch.equal(Jo, Jg.cpu())
    EB = random_fields(g, 9)
    Eg = EB.cuda()
    o.fill_ghosts(EB, True, 1, 5)
    ctx.fill_ghosts(Eg, True, 1, 5)
    torch.cuda.synchronize()
    assert torch.equal(EB, Eg.cpu())
    ctx.close()


class Padded(GridSpec):
    def strides(self):
        n1, n2, n3 = self.ext
        return (1, n1 + 3, (n1 + 3) * n2, (n1 + 3) * n2 * n3)


@pytest.mark.parametrize("n", [(40, 24, 1), (24, 20, 12)])
def test_padded_rows_and_six_species(n):
    """Rows of J longer than the grid's, and more species than one tiled
    launch takes, moving fast enough that some are left to the lists: the sums
    are exact, so J is the packed grid's bit for bit."""
    got = []
    for cls in (GridSpec, Padded):
        g = cls(dim=2 if n[2] == 1 else 3, n=n, order=2, real=torch.float32)
        ctx = Context(g)
        n1, n2, n3 = g.ext
        row = g.strides()[1]

        def field(src):
            f = torch.zeros((src.shape[0], n3, n2, row), device="cuda")
            f[..., :n1] = src.cuda()
            return f

        EB = random_fields(GridSpec(dim=g.dim, n=n, order=2, real=torch.float32), 5, amp=0.2)
        sp = []
        for k in range(6):
            s = make_species(g, 3, 2.0, 0.0, 50 + k, charge=(-1.0) ** k, index=k + 1).to("cuda")
            assert ctx.sort(s, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED) == abi.PIC_OK
            sp.append(s)
        Jg = torch.zeros((3, n3, n2, row), device="cuda")
        for _ in range(4):  # the binning goes stale: leavers are deferred
            Jg.zero_()
            ctx.push_deposit(sp, field(EB), Jg, 0.45, 0.7, g.dx)
        torch.cuda.synchronize()
        assert float(Jg[..., n1:].abs().sum()) == 0
        assert ctx.device_errors() == [0, 0, 0, 0]
        got.append((Jg[..., :n1].clone(), [torch.sort(s.u[0]).values for s in sp]))
        ctx.close()
    assert float(got[0][0].abs().max()) > 0
    assert torch.equal(got[0][0], got[1][0])
    assert all(torch.equal(a, b) for a, b in zip(got[0][1], got[1][1]))
