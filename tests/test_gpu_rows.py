"""Push and deposit by rows (16-byte words of the fields and currents) against
the oracle: row alignments from odd extents, particles in the last rows of the
arrays, and arrays off a 16-byte boundary, which keep the scalar path."""
import pytest
import torch

from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from oracle.oracle import Oracle
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


def _shifted(t, off):
    """A copy of t that starts `off` elements into its allocation."""
    flat = torch.zeros(t.numel() + off, dtype=t.dtype, device="cuda")
    v = flat[off:].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("dim,order", [(2, 1), (2, 2), (2, 3), (3, 1), (3, 2), (3, 3)])
@pytest.mark.parametrize("n1", [16, 17, 18, 19])
@pytest.mark.parametrize("off", [0, 1, 2])
def test_rows(dim, order, n1, off):
    g = GridSpec(dim=dim, n=(n1, 13, 11) if dim == 3 else (n1, 23, 1), order=order, real=torch.float32)
    o, ctx = Oracle(g), Context(g)
    EB = random_fields(g, 7 + n1, amp=0.2)
    s = make_species(g, 5, 0.4, 0.2, 3 * n1 + order)
    q = s.clone().to("cuda")
    Jo, Jg = empty_field(g, 3), _shifted(empty_field(g, 3), off)
    o.push(s, EB, 0.45, 0.6, g.dx)
    o.deposit([s], Jo, 0.45, g.dx)
    EBg = _shifted(EB, off)
    ctx.push(q, EBg, 0.45, 0.6, g.dx)
    ctx.deposit([q], Jg, 0.45, g.dx)
    torch.cuda.synchronize()
    for a, b in zip(s.i[:dim] + s.dx[:dim] + s.u, q.i[:dim] + q.dx[:dim] + q.u):
        assert torch.equal(a, b.cpu())
    # summation order: the bound of every deposit against the oracle
    assert float((Jo - Jg.cpu()).abs().max()) <= 4e-6 * float(Jo.abs().max())
    assert ctx.device_errors() == [0, 0, 0, 0]


@pytest.mark.parametrize("order", [1, 2, 3])
def test_single_particle_rows_are_exact(order):
    """One particle: every entry of J is one contribution, the oracle's bits,
    and the nodes around its rows stay zero."""
    g = GridSpec(dim=3, n=(17, 14, 12), order=order, real=torch.float32)
    EB = random_fields(g, 2, amp=0.3)
    for seed in range(40):
        o, ctx = Oracle(g), Context(g)
        s = make_species(GridSpec(dim=3, n=(1, 1, 1), order=order, real=torch.float32, ng=1), 1, 0.8, 0.0, seed)
        gen = torch.Generator().manual_seed(seed)
        for d in range(3):
            s.i[d] = torch.randint(0, g.n[d], (1,), generator=gen, dtype=torch.int32)
        q = s.clone().to("cuda")
        Jo, Jg = empty_field(g, 3), empty_field(g, 3, "cuda")
        o.push(s, EB, 0.45, 0.6, g.dx)
        o.deposit([s], Jo, 0.45, g.dx)
        ctx.push(q, EB.cuda(), 0.45, 0.6, g.dx)
        ctx.deposit([q], Jg, 0.45, g.dx)
        torch.cuda.synchronize()
        assert torch.equal(Jo, Jg.cpu()), seed
        ctx.close()
