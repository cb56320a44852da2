"""The record sort against a stable host sort, at the edges of its blocks (256
and 2048 particles), of its bins (one, about a thousand, more than 1024
particles in a cell) and of its layouts."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, make_species
from entity_gb300.sim import Context

pytestmark = pytest.mark.gpu


def _species(g, n, span, dead, seed):
    s = make_species(GridSpec(dim=g.dim, n=(n, 1, 1), order=2, real=g.real), 1, 0.1, 0.0, seed)
    gen = torch.Generator().manual_seed(seed)
    for d in range(3):
        hi = min(span, g.n[d]) if d < g.dim else 1
        s.i[d] = torch.randint(0, hi, (n,), generator=gen, dtype=torch.int32)
        s.dx[d] = torch.rand(n, generator=gen) if d < g.dim else torch.zeros(n)
        s.i_prev[d] = torch.randint(0, 9, (n,), generator=gen, dtype=torch.int32)
        s.dx_prev[d] = torch.rand(n, generator=gen)
    s.w = torch.rand(n, generator=gen).to(g.real)
    s.tag[torch.rand(n, generator=gen) < dead] = 0
    s.phi = torch.rand(n, generator=gen).to(g.real)
    return s


def _arrays(s, dim, prev):
    out = s.i[:dim] + s.dx[:dim] + s.u + [s.w, s.tag]
    return out + (s.i_prev[:dim] + s.dx_prev[:dim] if prev else [])


@pytest.mark.parametrize("dim,real,prev,extra", [
    (2, torch.float32, False, False), (2, torch.float64, True, False), (3, torch.float32, True, True),
    (3, torch.float32, False, False), (3, torch.float64, False, True), (3, torch.float64, True, False),
    (2, torch.float32, True, True), (2, torch.float64, False, False)])
@pytest.mark.parametrize("span,dead", [(64, 0.0), (2, 0.2), (1, 0.0), (1, 0.9)])
def test_record_sort_matches_host(dim, real, prev, extra, span, dead):
    g = GridSpec(dim=dim, n=(20, 18, 12) if dim == 3 else (40, 30, 1), order=2, real=real)
    for n in (1, 255, 256, 257, 1024, 1025, 2047, 2049, 6001):
        s = _species(g, n, span, dead, 7 * n + dim)
        if not extra:
            s.phi = None
        alive = s.tag == 1
        for flags in (abi.PIC_SORT_SPATIAL, abi.PIC_SORT_REMOVE_DEAD,
                      abi.PIC_SORT_SPATIAL | abi.PIC_SORT_REMOVE_DEAD):
            cells = 1
            key = torch.zeros(n, dtype=torch.int64)
            if flags & abi.PIC_SORT_SPATIAL:
                for d in range(dim):
                    key = key * g.n[d] + s.i[d].long()
                    cells *= g.n[d]
            key[~alive] = cells
            order = torch.sort(key, stable=True).indices
            ctx = Context(g)
            q = s.clone().to("cuda")
            assert ctx.sort(q, flags | (0 if prev else abi.PIC_SORT_SKIP_PREV)) == abi.PIC_OK
            want = [x[order] for x in _arrays(s, dim, prev)]
            for x, y in zip(want, _arrays(q, dim, prev)):
                assert torch.equal(x, y.cpu()), (n, flags)
            if extra:
                assert torch.equal(s.phi[order], q.phi.cpu())
            assert q.npart == (int(alive.sum()) if flags & abi.PIC_SORT_REMOVE_DEAD else n)
            ctx.close()
