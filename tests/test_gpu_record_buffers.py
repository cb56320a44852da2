"""The tiled kernel's record buffers: a context that found no memory for them
uses them once there is some, and their first use from two streams at once."""
import ctypes as C

import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from entity_gb300.sim import make_species as mk
from tests.helpers import random_fields

pytestmark = pytest.mark.gpu


def _plasma(g, ppc, seed):
    out = []
    ctx = Context(g)
    for k, q in enumerate((-1.0, 1.0)):
        s = make_species(g, ppc, 0.5, 0.0, seed + k, charge=q, index=k + 1, device="cuda")
        assert ctx.sort(s, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED) == abi.PIC_OK
        out.append(s)
    return ctx, out


def _call(g, ctx, sp, EB):
    here, J = [s.clone() for s in sp], empty_field(g, 3, "cuda")
    ctx.push_deposit(here, EB, J, 0.3, 0.5, g.dx)
    torch.cuda.synchronize()
    return J, here


def test_buffers_are_asked_for_again():
    """3D order 3: 36 x 1024 records of 32 bytes, two regions, for every SM: over
    350 MB. The first call finds 300 MB free, the second all of it."""
    g = GridSpec(dim=3, n=(32, 32, 32), order=3, real=torch.float32)
    EB = random_fields(g, 5, amp=0.1).cuda()
    first, sp = _plasma(g, 4, 31)
    want, parts = _call(g, first, sp, EB)  # (loads the kernels)
    first.close()
    ctx, sp = _plasma(g, 4, 31)
    small = empty_field(g, 3, "cuda")
    ctx.push_deposit([], EB, small, 0.3, 0.5, g.dx)  # (the exact accumulator)
    torch.cuda.empty_cache()
    spare = [torch.empty(64 << 20, dtype=torch.uint8, device="cuda")]  # what the calls clone
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (300 << 20), dtype=torch.uint8, device="cuda")
    del spare
    J, here = _call(g, ctx, sp, EB)
    assert torch.equal(J, want)
    for a, b in zip(here, parts):
        assert all(torch.equal(x, y) for x, y in zip(a.i + a.dx + a.u, b.i + b.dx + b.u))
    del hog, here
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    J2, here = _call(g, ctx, sp, EB)
    assert torch.equal(J2, want)
    assert before - torch.cuda.mem_get_info()[0] > (330 << 20)
    assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
    ctx.close()


@pytest.mark.parametrize("dim,order,real", [(3, 2, torch.float32), (2, 2, torch.float32), (3, 1, torch.float64)])
def test_first_use_from_two_streams(dim, order, real):
    g = GridSpec(dim=dim, n=(64, 32, 32) if dim == 3 else (256, 128, 1), order=order, real=real)
    EB = random_fields(g, 5, amp=0.1).cuda()
    for attempt in range(4):
        ctx, sp = _plasma(g, 6, 50)
        ref = [s.clone() for s in sp]
        Js = [empty_field(g, 3, "cuda") for _ in range(4)]
        L, nt = abi.load(), C.c_int64(0)
        assert L.pic_tile_offsets(ctx.h, C.byref(mk(sp[0], dim)), None, 0, C.byref(nt), None) == abi.PIC_OK
        st = [torch.cuda.Stream() for _ in range(2)]

        def call(s, J, stream):
            assert L.pic_push_deposit_tiles(ctx.h, C.byref(mk(s, dim)), C.c_void_p(EB.data_ptr()),
                                            C.c_void_p(J.data_ptr()), 0.3, 0.5, g.dx, 0, nt.value, 0, stream) == abi.PIC_OK
        torch.cuda.synchronize()
        for k in range(2):  # a species to a stream: the context's first tiled launches
            call(sp[k], Js[k], C.c_void_p(st[k].cuda_stream))
        torch.cuda.synchronize()
        assert ctx.device_errors() == [0, 0, 0, 0] and ctx.wait_timeouts() == 0
        for k in range(2):
            call(ref[k], Js[2 + k], None)
        torch.cuda.synchronize()
        # float sums of the tiles' own totals, in any order: 8 tiles to an entry
        tol = 16 * (2.0 ** -24 if real == torch.float32 else 2.0 ** -53)
        for k in range(2):
            a, b = ref[k], sp[k]
            assert all(torch.equal(x, y) for x, y in zip(a.i[:dim] + a.dx[:dim] + a.u, b.i[:dim] + b.dx[:dim] + b.u))
            assert float((Js[k] - Js[2 + k]).abs().max()) <= tol * float(Js[2 + k].abs().max())
        ctx.close()
