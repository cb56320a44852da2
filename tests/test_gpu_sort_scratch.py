"""A sort that finds no memory for its packed records moves every array through the
permutation: the same order, in the same arrays."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, make_species
from entity_gb300.sim import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,real", [(3, torch.float32), (2, torch.float64)])
@pytest.mark.parametrize("tiled", [0, abi.PIC_SORT_TILED])
def test_sort_without_records(dim, real, tiled):
    """4.2 M particles: records of 64 bytes or more are 268 MB, the other way takes 84 MB
    and as much again of short-lived scan scratch; 200 MB are left free."""
    g = GridSpec(dim=dim, n=(64, 64, 64) if dim == 3 else (512, 512, 1), order=2, real=real)
    base = make_species(g, 16, 0.3, 0.0, 5, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(3)
    base.tag[torch.rand(base.npart, generator=gen, device="cuda") < 0.01] = 0
    flags = abi.PIC_SORT_SPATIAL | tiled
    got = []
    for hogged in (False, True):
        ctx, s = Context(g), base.clone()
        assert ctx.sort(make_species(g, 1, 0.1, 0.0, 6, device="cuda"), flags) == abi.PIC_OK  # (loads the kernels)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - (200 << 20), dtype=torch.uint8, device="cuda") if hogged else None
        assert ctx.sort(s, flags) == abi.PIC_OK
        torch.cuda.synchronize()
        del hog
        torch.cuda.empty_cache()
        got.append(s)
        assert ctx.device_errors() == [0, 0, 0, 0]
        ctx.close()
    a, b = got
    assert not torch.equal(a.i[0], base.i[0])
    for x, y in zip(a.i[:dim] + a.dx[:dim] + a.u + a.i_prev[:dim] + a.dx_prev[:dim] + [a.w, a.tag],
                    b.i[:dim] + b.dx[:dim] + b.u + b.i_prev[:dim] + b.dx_prev[:dim] + [b.w, b.tag]):
        assert torch.equal(x, y)
