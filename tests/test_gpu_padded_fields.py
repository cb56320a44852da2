"""Vector reductions and arrays with gaps: what lies between the elements of a padded
field stays as it is, and the sums are those of a packed one."""
import pytest
import torch

import entity_gb300.sim as sim
from entity_gb300.inputs import GridSpec, make_species
from entity_gb300.sim import Context, SpeciesAdjoint, step_params

pytestmark = pytest.mark.gpu
PAD = 3  # elements after a row


def _strides(g, pad):
    r = g.ext[0] + pad
    return (1, r, r * g.ext[1], r * g.ext[1] * g.ext[2])


def _field(g, ncomp, pad):
    """Zeros, the gaps holding the smallest denormal's bits."""
    f = torch.zeros(ncomp, g.ext[2], g.ext[1], g.ext[0] + pad, dtype=torch.float32, device="cuda")
    if pad:
        f.view(torch.int32)[..., g.ext[0]:] = 1
    return f


def _context(g, pad, monkeypatch):
    def grid(spec):
        p = sim_make_grid(spec)
        for k, s in enumerate(_strides(spec, pad)):
            p.em_stride[k] = p.cur_stride[k] = s
        return p
    sim_make_grid = sim.make_grid
    monkeypatch.setattr(sim, "make_grid", grid)
    ctx = Context(g)
    monkeypatch.setattr(sim, "make_grid", sim_make_grid)
    return ctx


def _gaps_untouched(g, f):
    return bool((f.view(torch.int32)[..., g.ext[0]:] == 1).all())


@pytest.mark.parametrize("dim,order", [(2, 2), (2, 3), (3, 1), (3, 2), (3, 3)])
def test_deposit_leaves_gaps_alone(dim, order, monkeypatch):
    g = GridSpec(dim=dim, n=(21, 18, 14) if dim == 3 else (37, 30, 1), order=order, real=torch.float32)
    got = []
    for pad in (0, PAD):
        ctx = _context(g, pad, monkeypatch)
        sp = make_species(g, 5, 0.5, 0.1, 7, device="cuda")
        EB, J = _field(g, 6, pad), _field(g, 3, pad)
        EB[..., :g.ext[0]] = 0.1
        ctx.push(sp, EB, 0.4, 0.5, g.dx)
        ctx.deposit([sp], J, 0.4, g.dx)
        F = _field(g, 3, pad)  # the fused call with float sums, by rows in 3D too
        ctx.push_deposit([sp], EB, F, 0.4, 0.5, g.dx, flags=4)
        torch.cuda.synchronize()
        if pad:
            assert _gaps_untouched(g, J) and _gaps_untouched(g, F)
        got.append([x[..., :g.ext[0]].double() for x in (J, F)])
        ctx.close()
    for a, b in zip(*got):
        # float sums in another order: up to 5 (order + 2)^dim additions of an entry
        n = 5 * (order + 2) ** dim
        assert float(a.abs().max()) > 0
        assert float((a - b).abs().max()) <= n * 2.0 ** -24 * float(a.abs().max())


@pytest.mark.parametrize("order", [1, 2, 3])
def test_adjoint_of_padded_fields(order, monkeypatch):
    g = GridSpec(dim=2, n=(37, 30, 1), order=order, real=torch.float32)
    prm = step_params(g, cfl=0.45, ppc0=8.0, skindepth0=10.0, larmor0=10.0)
    got = []
    for pad in (0, PAD):
        ctx = _context(g, pad, monkeypatch)
        sp = [make_species(g, 4, 0.01, 0.2, 7 + k, charge=(-1.0) ** k, index=k + 1, device="cuda") for k in range(2)]
        EB, J, buff, lam = (_field(g, c, pad) for c in (6, 3, 3, 6))
        EB[2, :, g.ng:-g.ng, g.ng:g.n[0] + g.ng] = 0.05
        adj = [SpeciesAdjoint(g, s.npart) for s in sp]
        loss = ctx.gradient(sp, adj, EB, J, buff, prm, 3, 2, lam)
        torch.cuda.synchronize()
        if pad:
            assert _gaps_untouched(g, EB)
        got.append((loss, lam[..., :g.ext[0]].double(), [x.double() for a in adj for x in a.lx + a.lu + [a.lw]]))
        ctx.close()
    (la, fa, pa), (lb, fb, pb) = got
    assert abs(la - lb) <= 1e-5 * abs(la)
    for a, b in zip([fa] + pa, [fb] + pb):
        assert float((a - b).abs().max()) <= 2e-3 * float(a.abs().max())
