"""A checkpoint that does not fit is refused before anything changes."""
import ctypes as C

import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, make_species
from entity_gb300.sim import Context
from entity_gb300.sim import make_species as mk
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", [0, 1])
def test_refused_restore_changes_nothing(small):
    g = GridSpec(dim=2, n=(16, 12, 1), order=2, real=torch.float32)
    ctx = Context(g)
    EB = random_fields(g, 5).cuda()
    sp = [make_species(g, 4, 0.2, 0.0, 3 + k, index=k + 1, device="cuda") for k in range(2)]
    ctx.checkpoint_save(0, sp, EB)
    torch.cuda.synchronize()
    other = [make_species(g, 4, 0.2, 0.0, 30 + k, index=k + 1, device="cuda") for k in range(2)]
    EB2 = random_fields(g, 6).cuda()
    arr = (abi.PicSpecies * 2)(*[mk(s, 2) for s in other])
    for k in range(2):
        arr[k].npart = 100 + k
    arr[small].maxnpart = 200
    keep = [[x.clone() for x in s.i + s.dx + s.u + [s.tag]] for s in other], EB2.clone()
    st = abi.load().pic_checkpoint_restore(ctx.h, 0, arr, 2, C.c_void_p(EB2.data_ptr()), None)
    torch.cuda.synchronize()
    assert st == abi.PIC_ERR_ARG
    assert [arr[k].npart for k in range(2)] == [100, 101]
    assert torch.equal(EB2, keep[1])
    for s, old in zip(other, keep[0]):
        assert all(torch.equal(a, b) for a, b in zip(s.i + s.dx + s.u + [s.tag], old))
    # and one that fits is restored
    arr[small].maxnpart = 0
    assert abi.load().pic_checkpoint_restore(ctx.h, 0, arr, 2, C.c_void_p(EB2.data_ptr()), None) == abi.PIC_OK
    torch.cuda.synchronize()
    assert torch.equal(EB2, EB) and arr[0].npart == sp[0].npart
    assert all(torch.equal(a, b) for a, b in zip(other[1].u, sp[1].u))
    ctx.close()
