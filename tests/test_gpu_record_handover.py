"""Record buffers passed from CTA to CTA: more tiles than buffers, and launches
back to back, so that every buffer changes hands many times."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


# tiles of 16 x 8 (x 8) cells in FP32, 8 x 8 x 4 in 3D FP64 and 8^3 at order 3
@pytest.mark.parametrize("n,order,real", [
    ((160, 64, 64), 2, torch.float32), ((96, 64, 64), 3, torch.float32), ((64, 64, 40), 2, torch.float64),
    ((512, 512, 1), 1, torch.float32)])
def test_buffers_change_hands(n, order, real, monkeypatch):
    """J of each of eight unsynchronised calls against the same call without
    records: the same bits in FP32 (integer sums); in FP64 each tile's integer
    sums are rounded to the same doubles, and the up to 8 tiles that share an
    entry add theirs in any order: 8 * 2^-53 of the largest."""
    dim = 2 if n[2] == 1 else 3
    g = GridSpec(dim=dim, n=n, order=order, real=real)
    EB = random_fields(g, 5, amp=0.1).cuda()
    ctx = Context(g)
    sp = []
    for k, q in enumerate((-1.0, 1.0)):
        s = make_species(g, 4, 1.0, 0.0, 41 + k, charge=q, index=k + 1, device="cuda")
        assert ctx.sort(s, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED) == abi.PIC_OK
        sp.append(s)
    got = []
    for off in ("0", "1"):
        monkeypatch.setenv("ENTITY_PIC_NO_RECORDS", off)
        here, Js = [s.clone() for s in sp], []
        for _ in range(8):
            Js.append(empty_field(g, 3, "cuda"))
            ctx.push_deposit(here, EB, Js[-1], 0.2, 0.7, g.dx)
        torch.cuda.synchronize()
        got.append((Js, here))
    for a, b in zip(*(x[0] for x in got)):
        top = float(b.abs().max())
        assert top > 0
        if real == torch.float32:
            assert torch.equal(a, b)
        else:
            assert float((a - b).abs().max()) <= 8 * 2.0 ** -53 * top
    for a, b in zip(*(x[1] for x in got)):
        assert all(torch.equal(p, q) for p, q in zip(a.i[:dim] + a.dx[:dim] + a.u, b.i[:dim] + b.dx[:dim] + b.u))
    assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
    ctx.close()
