"""Checkpoint slots: many arrays copied in one launch, at sizes and offsets off
the 16-byte boundary, with more arrays than one launch takes, and a slot reused
for fewer and for more particles. Bytes are bytes: equality."""
import pytest
import torch

from entity_gb300.inputs import GridSpec, make_species
from entity_gb300.sim import Context
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


def _species(g, n, seed, off):
    s = make_species(GridSpec(dim=g.dim, n=(max(n, 4) + off, 1, 1), order=g.order, real=g.real), 1, 0.4, 0.0, seed)
    gen = torch.Generator().manual_seed(seed)
    for d in range(3):
        s.i[d] = torch.randint(0, g.n[d], (n + off,), generator=gen, dtype=torch.int32)
        s.dx[d] = torch.rand(n + off, generator=gen)
        s.u[d] = torch.rand(n + off, generator=gen, dtype=torch.float64).to(g.real)
    s.w, s.tag = torch.ones(n + off, dtype=g.real), torch.randint(0, 2, (n + off,), generator=gen).to(torch.int16)
    s.i_prev, s.dx_prev = [x.clone() for x in s.i], [x.clone() for x in s.dx]
    s = s.clone().to("cuda")
    cut = lambda v: [x[off:] for x in v]  # views that start off the 16-byte boundary
    s.i, s.dx, s.u, s.i_prev, s.dx_prev = cut(s.i), cut(s.dx), cut(s.u), cut(s.i_prev), cut(s.dx_prev)
    s.w, s.tag, s.npart = s.w[off:], s.tag[off:], n
    return s


def _state(g, s):
    n = s.npart
    return [t[:n].clone() for t in s.i[:g.dim] + s.dx[:g.dim] + s.u + [s.tag]]


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("off", [0, 1, 3])
def test_slots(dim, real, off):
    g = GridSpec(dim=dim, n=(9, 7, 1 if dim == 2 else 5), order=1, real=real)
    ctx = Context(g)
    EB = random_fields(g, 3).cuda()
    # four species: 4 (2 dim + 4) + 1 arrays, more than one launch
    for sizes in ((5, 8, 1, 4097), (300001, 64, 63, 2), (7, 100, 65536, 31)):
        sp = [_species(g, n, 10 + k, off) for k, n in enumerate(sizes)]
        want, eb = [_state(g, s) for s in sp], EB.clone()
        ctx.checkpoint_save(1, sp, EB)
        for s in sp:
            for t in s.i[:dim] + s.dx[:dim] + s.u + [s.tag]:
                t.zero_()
        EB.zero_()
        ctx.checkpoint_restore(1, sp, EB)
        torch.cuda.synchronize()
        assert torch.equal(EB, eb)
        for s, w in zip(sp, want):
            assert all(torch.equal(a, b) for a, b in zip(_state(g, s), w))
    ctx.close()
