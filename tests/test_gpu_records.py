"""Deposit records of the tiled kernel at the edges of their queues: chunks of
particles that just fit, or not, between two deposits, and a bank class that
overflows into the others because every particle starts in one cell."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu

# particles of one tile between two deposits (TileShape::CHUNK)
CHUNK = {(3, torch.float32): 20480, (3, torch.float64): 4608, (2, torch.float32): 2048,
         (2, torch.float64): 2048}


def _one_tile(g, n, one_cell, temp, seed):
    """n particles of each of two species in the first tile of the grid, all
    in one cell or spread over the tile's 8 x 8 (x 4) corner."""
    out = []
    for k, q in enumerate((-1.0, 1.0)):
        s = make_species(GridSpec(dim=g.dim, n=(n, 1, 1), order=g.order, real=g.real), 1, temp, 0.0,
                         seed + k, charge=q, index=k + 1)
        gen = torch.Generator().manual_seed(seed + 10 + k)
        for d in range(g.dim):
            hi = 1 if one_cell else (8, 8, 4)[d]
            s.i[d] = torch.randint(0, hi, (n,), generator=gen, dtype=torch.int32) + 3 * one_cell
            s.dx[d] = torch.rand(n, generator=gen, dtype=torch.float32)
        if g.dim == 2:
            s.i[2], s.dx[2] = torch.zeros(n, dtype=torch.int32), torch.zeros(n)
        s.i_prev, s.dx_prev = [x.clone() for x in s.i], [x.clone() for x in s.dx]
        out.append(s)
    return out


@pytest.mark.parametrize("one_cell", [False, True])
@pytest.mark.parametrize("dim,order,real", [
    (3, 1, torch.float32), (3, 2, torch.float32), (3, 3, torch.float32), (2, 1, torch.float32),
    (2, 2, torch.float32), (2, 3, torch.float32), (3, 2, torch.float64), (2, 2, torch.float64)])
def test_records_at_chunk_edges(dim, order, real, one_cell, monkeypatch):
    """J from records against J with every particle deposited as it is pushed:
    the same bits in FP32 (integer sums); in FP64 each entry is rounded once
    at the flush from the same integer totals, and the flush's double atomics
    add at most 8 tiles' values: 8 * 2^-53 of the largest, 1e-15."""
    n3 = (32, 32, 16) if dim == 3 else (64, 32, 1)
    g = GridSpec(dim=dim, n=n3, order=order, real=real)
    EB = random_fields(g, 5, amp=0.1).cuda()
    c = 36864 if (dim, order, real) == (3, 3, torch.float32) else CHUNK[dim, real]
    for n in (1, 33, c // 2 - 1, c // 2 + 1, c + 17):
        ctx = Context(g)
        gpu = [s.to("cuda") for s in _one_tile(g, n, one_cell, 0.5, 100 + n)]
        for s in gpu:
            assert ctx.sort(s, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED) == abi.PIC_OK
        got = []
        for off in ("0", "1"):
            monkeypatch.setenv("ENTITY_PIC_NO_RECORDS", off)
            sp = [s.clone() for s in gpu]
            J = empty_field(g, 3, "cuda")
            ctx.push_deposit(sp, EB, J, 0.45, 0.7, g.dx)
            torch.cuda.synchronize()
            got.append((J, sp))
        (Ja, a), (Jb, b) = got
        assert float(Jb.abs().max()) > 0
        if real == torch.float32:
            assert torch.equal(Ja, Jb), n
        else:
            assert float((Ja - Jb).abs().max()) <= 1e-15 * float(Jb.abs().max()), n
        for x, y in zip(a, b):
            assert all(torch.equal(p, q) for p, q in zip(x.i + x.dx + x.u, y.i + y.dx + y.u))
        assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
        ctx.close()
