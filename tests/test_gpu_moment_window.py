"""The windowed moment deposit against the oracle: particle orders that the
shared window holds, does not hold, or holds in part, remainders of its chunks
of 4096 particles, and coefficients that the fixed-point scale cannot take."""
import pytest
import torch

from entity_gb300 import abi
from entity_gb300.inputs import GridSpec, empty_field, make_species
from entity_gb300.sim import Context
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _species(g, n, layout, weight, seed):
    s = make_species(GridSpec(dim=g.dim, n=(n, 1, 1), order=2, real=g.real), 1, 0.3, 0.0, seed,
                     with_prev=False)
    gen = torch.Generator().manual_seed(seed)
    for d in range(g.dim):
        m = g.n[d]
        r = torch.randint(0, m, (n,), generator=gen, dtype=torch.int32)
        if layout == "cell":
            r = torch.full((n,), m - 1, dtype=torch.int32)
        elif layout == "clump":  # most in a corner, some across the periodic edge
            r = torch.where(torch.rand(n, generator=gen) < 0.03, r, r % 6)
        s.i[d] = r
        s.dx[d] = torch.rand(n, generator=gen)
    for d in range(g.dim, 3):
        s.i[d], s.dx[d] = torch.zeros(n, dtype=torch.int32), torch.zeros(n)
    s.w = (weight * (0.5 + torch.rand(n, generator=gen, dtype=torch.float64))).to(g.real)
    s.tag[torch.rand(n, generator=gen) < 0.1] = 0
    return s


# the bound of test_gpu_output: summation order, of the largest cell
@pytest.mark.parametrize("dim,real,tol", [(2, torch.float32, 2e-5), (3, torch.float32, 2e-5),
                                          (2, torch.float64, 1e-12), (3, torch.float64, 1e-12)])
@pytest.mark.parametrize("layout", ["random", "clump", "cell"])
@pytest.mark.parametrize("weight,spread", [(1.0, 1.0), (1e-30, 1.0), (1e30, 1.0), (1.0, 1e-6)])
def test_moment_window(dim, real, tol, layout, weight, spread):
    g = GridSpec(dim=dim, n=(70, 61, 1) if dim == 2 else (40, 33, 36), order=3, real=real)
    o, ctx = Oracle(g), Context(g)
    for n, order in ((1, 2), (4095, 1), (4097, 0), (9001, 2), (5000, 3), (4500, 5)):
        s = _species(g, n, layout, weight, n)
        s.tag[0] = 1
        s.w[::2] *= spread
        for smoothing in (abi.PIC_SMOOTH_SPLINE, abi.PIC_SMOOTH_CONST):
            d = dict(id=abi.PIC_MOM_T, c1=0, c2=1, order=order, smoothing=smoothing, use_weights=1,
                     inv_n0=0.5, dx=0.75)
            p = abi.PicMomentParams()
            for k, v in d.items():
                setattr(p, k, v)
            a, b = empty_field(g, 6), empty_field(g, 6, "cuda")
            o.output_moment([s], d, a, 3)
            ctx.output_moment([s.to("cuda")], p, b, 3)
            torch.cuda.synchronize()
            scale = float(a.double().abs().max())
            assert scale > 0
            assert float((a.double() - b.cpu().double()).abs().max()) <= tol * scale, (n, order)
    assert ctx.device_errors() == [0, 0, 0, 0]
