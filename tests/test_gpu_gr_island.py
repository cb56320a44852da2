"""The FP64 island's push (its own formulas on the device) and the early end of
the geodesic passes, against the oracle's double-precision push of the same
FP32 particles; the GR field kernels at the remainders of their rows."""
import pytest
import torch

from tests.test_gpu_gr import TOL, _particles, _rand_fields, _setup, _X

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


@pytest.mark.parametrize("real", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [(4, 8), (29, 9), (30, 16), (31, 12), (61, 10), (128, 24)])
def test_field_rows(n, real):
    """The field kernels' rows of 30 and 32 cells, one and several per warp, at
    their remainders, against the oracle."""
    from entity_gb300.inputs import empty_field
    g, spec, ctx, o = _setup(real, order=2, n=n)
    em, J = _rand_fields(g, 3), _rand_fields(g, 4)[:3].clone()
    emg, Jg = em.cuda(), J.cuda()

    def same(a, b, what):  # the bound of the field kernels' parity (test_gpu_gr)
        torch.cuda.synchronize()
        assert float((a - b.cpu()).abs().max()) <= 10 * TOL[real] * float(a.abs().max()), what

    for which, ref in enumerate((o.gr_aux_e, o.gr_aux_h)):
        a, b = empty_field(g, 6), empty_field(g, 6, "cuda")
        ref(em, em, a)
        ctx.gr_aux(which, emg, emg, b)
        same(a, b, which)
    for name in ("gr_faraday", "gr_ampere"):
        a, b = em.clone(), emg.clone()
        getattr(o, name)(em, a, em, 0.01)
        getattr(ctx, name)(emg, b, emg, 0.01)
        same(a, b, name)
    a, b = em.clone(), emg.clone()
    o.gr_currents_ampere(a, J, 0.01)
    ctx.gr_currents_ampere(b, Jg, 0.01)
    same(a, b, "currents")
