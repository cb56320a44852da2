"""The FP64 island's push (its own formulas on the device) and the early end of
the geodesic passes, against the oracle's double-precision push of the same
FP32 particles."""
import pytest
import torch

from tests.test_gpu_gr import _particles, _rand_fields, _setup, _X

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2, 3])
@pytest.mark.parametrize("h", [0.0, 0.25])
@pytest.mark.parametrize("pusher,dt,niter", [(1, 0.05, 10), (1, 1e-4, 10), (1, 0.5, 3), (3, 0.05, 10),
                                             (3, 1e-4, 1)])
def test_island_push(order, h, pusher, dt, niter):
    """Both sides push in double from the same FP32 values and round once: the
    double results differ by some 1e-13, the rounded ones by an ulp (2^-23 of
    the largest u; 2^-18 of X below 64)."""
    g, spec, ctx, o = _setup(torch.float32, order=order, h=h)
    em, em0 = _rand_fields(g, 1), _rand_fields(g, 2)
    sp = _particles(g, 4000, 5, pusher=pusher)
    sp.i[1][:400], sp.i[1][400:800] = 0, g.n[1] - 1  # beside the axes
    spg = sp.clone().to("cuda")
    o.gr_push(sp, em, em0, dt, 2.0, niter, island=(0, g.n[0]))
    ctx.gr_push(spg, em.cuda(), em0.cuda(), dt, 2.0, niter, island=(0, g.n[0]))
    torch.cuda.synchronize()
    assert ctx.device_errors() == [0, 0, 0, 0]
    assert torch.equal(sp.tag, spg.tag.cpu())
    ok = sp.tag == 1
    for d in range(2):
        assert float((_X(sp, d) - _X(spg, d))[ok].abs().max()) <= 2.0 ** -17
    for c in range(3):
        a, b = sp.u[c].double()[ok], spg.u[c].cpu().double()[ok]
        assert bool(torch.isfinite(a).all())
        assert float((a - b).abs().max()) <= 2.0 ** -22 * float(a.abs().max())
