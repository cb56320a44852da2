"""The workloads whose time is watched, through the package's public entry points.

Each case is a call (or the short sequence of calls) that a program using this library makes over and
over: a step of an engine, the reference's own order of phase calls, a start-up, an output, a gradient.
Sizes follow bench.py's workloads (the 512^2 pair plasma, the 256^3 turbulence box, the order-3
magnetised plasma, the two-stream gradient, the Wald problem, the output preparation) and small, odd
and ragged boxes around them.

`exact` restates the special-relativistic step, the injection-free part of the output and the gradient
with torch in 64 bits (cardinal B-spline shapes, Esirkepov's deposit, the Yee solver, autograd).
"""
import math

import torch

from entity_gb300 import abi
from entity_gb300.inputs import (GridSpec, empty_field, empty_species, inject_params,
                                 make_species)
from entity_gb300.sim import Context, SpeciesAdjoint, step_params

STEP3D = dict(kind="step", dim=3, order=2, real="f32", ppc=8, temp=0.09, drift=0.0, B0=0.1, dB=1.0, dE=0.05,
              nfilter=4, sort=8)
STEP2D = dict(kind="step", dim=2, n3=1, order=1, real="f32", ppc=16, temp=0.01, drift=0.3, B0=0.1, dB=0.0,
              dE=0.02, nfilter=0, sort=16)


def listed():
    return [
        # a test-sized 2D box, as used while a set-up is being written: launches and host work count
        dict(STEP2D, name="pair2d_64", n1=64, n2=64),
        # the 2D pair plasma of the benchmark: drifting beams, 16 ppc each, order 1
        dict(STEP2D, name="pair2d_512", n1=512, n2=512),
        # a 2D shock- or reconnection-like box of odd sizes, order 2, filtered currents, few particles per cell
        dict(STEP2D, name="ragged2d", n1=777, n2=333, order=2, ppc=9, temp=0.1, drift=0.0, dB=0.5, nfilter=2,
             sort=10),
        # a small ragged 3D turbulence box, as one domain of a decomposed run has it
        dict(STEP3D, name="ragged3d", n1=100, n2=75, n3=61),
        # the 3D decaying turbulence of the benchmark at full size: 268 M particles
        dict(STEP3D, name="turb3d_256", n1=256, n2=256, n3=256),
        # the order-3 magnetised plasma (sigma 10, theta 1, 32 ppc each) on a quarter of its box
        dict(STEP3D, name="sweep3d_96", n1=96, n2=96, n3=96, order=3, ppc=32, temp=1.0, B0=0.3162, dB=0.0,
             nfilter=0, sort=4),
        # double precision, the reference's precision=double build: the turbulence box of the precision study
        dict(STEP3D, name="turb3d_f64", n1=64, n2=64, n3=64, real="f64"),
        # the reference's phase order with separate push and deposit calls, previous positions stored, and no
        # spatial sort (its default): particles in injection order, which is random
        dict(STEP3D, name="phases3d", kind="phases", n1=96, n2=96, n3=96, nfilter=2),
        # start-up or continuous injection: pairs drawn into both species, then the spatial sort of each
        dict(name="populate3d", kind="populate", dim=3, n1=128, n2=128, n3=128, order=2, real="f32", ppc=8,
             temp=0.09),
        # an output step: density and energy-density moments, the electric field, every tenth particle
        dict(STEP3D, name="output3d", kind="output", n1=128, n2=128, n3=128, mom_order=2),
        # general relativity: the Wald problem around a Kerr black hole
        dict(name="wald2d", kind="wald", n1=1024, n2=512, order=2, real="f32", ppc=4, a=0.95),
        # the gradient of the final field energy of a two-stream plasma through checkpointed steps
        dict(name="gradient2d", kind="gradient", dim=2, n1=256, n2=256, n3=1, order=2, real="f32", ppc=16,
             temp=1e-4, drift=0.2, steps=32, every=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step2d", "step2d", "step3d", "step3d", "step3d", "phases", "populate", "output", "wald",
                       "gradient"])
    if kind == "step2d":
        n1, n2 = _log(rng, 48, 1200), _log(rng, 48, 1200)
        return dict(STEP2D, n1=n1, n2=n2, order=rng.choice([1, 1, 2, 3]), ppc=rng.randint(4, 32),
                    temp=rng.choice([0.01, 0.1, 1.0]), drift=rng.choice([0.0, 0.3]), dB=rng.choice([0.0, 0.5]),
                    nfilter=rng.randint(0, 4), sort=rng.choice([8, 10, 16]),
                    real=rng.choice(["f32", "f32", "f32", "f64"]))
    if kind == "step3d":
        real = rng.choice(["f32", "f32", "f32", "f64"])
        hi = 180 if real == "f32" else 72
        n = [_log(rng, 24, hi) for _ in range(3)]
        return dict(STEP3D, n1=n[0], n2=n[1], n3=n[2], order=rng.choice([1, 2, 2, 3]), ppc=rng.randint(4, 24),
                    temp=rng.choice([0.01, 0.09, 1.0]), nfilter=rng.randint(0, 4), sort=rng.choice([4, 8]),
                    real=real)
    if kind == "phases":
        n = [_log(rng, 24, 110) for _ in range(3)]
        return dict(STEP3D, kind=kind, n1=n[0], n2=n[1], n3=n[2], order=rng.choice([1, 2, 2, 3]),
                    ppc=rng.randint(3, 10), nfilter=rng.randint(0, 4))
    if kind == "populate":
        dim = rng.choice([2, 3])
        n = [_log(rng, 32, 150) for _ in range(3)] if dim == 3 else [_log(rng, 64, 1200), _log(rng, 64, 1200), 1]
        return dict(kind=kind, dim=dim, n1=n[0], n2=n[1], n3=n[2], order=2, real="f32", ppc=rng.randint(3, 12),
                    temp=rng.choice([0.0, 0.09, 1.0]))
    if kind == "output":
        n = [_log(rng, 32, 150) for _ in range(3)]
        return dict(STEP3D, kind=kind, n1=n[0], n2=n[1], n3=n[2], ppc=rng.randint(3, 12),
                    mom_order=rng.choice([0, 1, 2, 3]))
    if kind == "wald":
        return dict(kind=kind, n1=_log(rng, 200, 1100), n2=_log(rng, 100, 560), order=2, real="f32",
                    ppc=rng.randint(2, 5), a=rng.choice([0.6, 0.8, 0.95]))
    return dict(kind="gradient", dim=2, n1=_log(rng, 64, 300), n2=_log(rng, 64, 300), n3=1, order=rng.choice([2, 3]),
                real="f32", ppc=rng.randint(6, 18), temp=1e-4, drift=0.2, steps=rng.randint(12, 32),
                every=rng.choice([4, 6, 8]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _grid(c):
    return GridSpec(dim=c["dim"], n=(c["n1"], c["n2"], c["n3"]), order=c["order"],
                    real=torch.float32 if c["real"] == "f32" else torch.float64)


def _modes(g, B0, dB, dE, seed):
    """EB = B0 along x3 plus 8 long-wave modes in every component, ghosts holding the periodic images."""
    gen = torch.Generator().manual_seed(seed)
    EB = empty_field(g, 6, "cuda")
    ax = []
    for d in range(3):
        N = (g.ext[2 - d])
        ng = g.ng if N > 1 else 0
        ax.append(((torch.arange(N, device="cuda", dtype=torch.float64) - ng) / g.n[2 - d]) * 2 * math.pi)
    for comp in range(6):
        amp = dE * B0 if comp < 3 else dB * B0
        v = torch.zeros(EB.shape[1:], dtype=torch.float64, device="cuda")
        for _ in range(4 if amp else 0):
            k = torch.randint(-2, 3, (3,), generator=gen).tolist()
            ph = 2 * math.pi * float(torch.rand((), generator=gen))
            arg = (k[0] * ax[0])[:, None, None] + (k[1] * ax[1])[None, :, None] + (k[2] * ax[2])[None, None, :]
            v += amp * 0.5 * torch.cos(arg + ph)
        EB[comp] = (v + (B0 if comp == 5 else 0.0)).to(g.real)
    return EB


def _pair(c, g, seed, shuffle, with_prev, weights=None):
    out = []
    for k, q in enumerate((-1.0, 1.0)):
        out.append(make_species(g, c["ppc"], c["temp"], c["drift"] * (1 if k == 0 else -1), 2 * seed + 11 + k,
                                charge=q, index=k + 1, device="cuda", shuffle=shuffle, with_prev=with_prev,
                                weights=weights))
    return out


def _params(c, g):
    return step_params(g, cfl=0.45, ppc0=2.0 * c["ppc"], skindepth0=10.0, larmor0=1.0 / c["B0"],
                       nfilter=c["nfilter"], sort_interval=c["sort"], write_prev=False, sort_tiled=True)


class State:
    pass


def prepare(case, seed):
    c, s = case, State()
    s.c = c
    if c["kind"] == "wald":
        from entity_gb300.gr import gr_step_params, horizon_island, wald_setup
        g, spec, s.ctx, s.fields, s.sp = wald_setup(n=(c["n1"], c["n2"]), a=c["a"], order=c["order"],
                                                    ppc=c["ppc"], seed=seed + 1)
        s.prm = gr_step_params(s.ctx, cfl=0.5, ppc0=2.0, skindepth0=0.05, larmor0=0.0025)
        s.island, s.k = horizon_island(g, spec), 1
        # step 0 brings the leapfrog's fields to their starting times
        s.ctx.grpic_step(s.sp, s.fields, s.prm, island=s.island, step=0, match=s.ctx.match)
        return s
    g = s.g = _grid(c)
    s.ctx = Context(g)
    if c["kind"] == "populate":
        cap = g.ncells() * c["ppc"]
        s.sp = [empty_species(g, cap, charge=q, index=k + 1) for k, q in enumerate((-1.0, 1.0))]
        s.inj = inject_params(1.0, 2.0 * c["ppc"], [(0, g.n[d]) for d in range(g.dim)], (c["temp"], c["temp"]),
                              seed=seed + 1)
        return s
    if c["kind"] == "gradient":
        gen = torch.Generator().manual_seed(seed)
        ph = 2 * math.pi * float(torch.rand((), generator=gen))
        k = 2 * math.pi / g.n[0]
        s.sp = _pair(c, g, seed, False, False,
                     weights=lambda i, d: 1.0 + 0.05 * torch.cos(k * (i[0].double() + d[0].double()) + ph))
        s.EB = _modes(g, 0.1, 0.0, 0.1, seed)
        s.EB[3:] = 0.0
        s.prm = step_params(g, cfl=0.45, ppc0=2.0 * c["ppc"], skindepth0=10.0, larmor0=10.0)
        s.J, s.buff, s.lam = empty_field(g, 3, "cuda"), empty_field(g, 3, "cuda"), empty_field(g, 6, "cuda")
        s.adj = [SpeciesAdjoint(g, x.npart) for x in s.sp]
        return s
    s.EB = _modes(g, c["B0"], c["dB"], c["dE"], seed)
    s.J, s.buff = empty_field(g, 3, "cuda"), empty_field(g, 3, "cuda")
    s.prm = _params(c, g)
    phases = c["kind"] == "phases"
    s.sp = _pair(c, g, seed, phases, phases)
    s.k = 1
    if not phases:  # a run in progress: the species were sorted a step ago
        for x in s.sp:
            s.ctx.sort(x, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED | abi.PIC_SORT_SKIP_PREV)
    if c["kind"] == "output":
        s.mom, s.out = empty_field(g, 6, "cuda"), torch.empty((3,) + tuple(reversed(g.n)), dtype=g.real, device="cuda")
        n = s.sp[0].npart // 10
        s.rec = [torch.empty(n, dtype=g.real, device="cuda") for _ in range(7)]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _moment(c, g, mid, c1=0, c2=0):
    p = abi.PicMomentParams()
    p.id, p.c1, p.c2, p.order, p.smoothing = mid, c1, c2, c["mom_order"], abi.PIC_SMOOTH_SPLINE
    p.use_weights, p.inv_n0, p.dx = 1, 1.0 / (2.0 * c["ppc"]), g.dx
    return p


def _particles(s, more=()):
    D = s.c.get("dim", 2)
    return [dict(i=x.i[:D], dx=x.dx[:D], u=x.u, **{m: getattr(x, m) for m in more}) for x in s.sp]


def run(s):
    c = s.c
    if c["kind"] == "step":
        s.ctx.step(s.sp, s.EB, s.J, s.buff, s.prm, s.k)
        s.k += 1
        return dict(EB=s.EB, J=s.J, sp=_particles(s))
    if c["kind"] == "phases":
        p, g = s.prm, s.g
        for x in s.sp:
            s.ctx.push(x, s.EB, p.dt, p.omegaB0, p.dx)
        s.ctx.deposit(s.sp, s.J, p.dt, p.dx)
        s.ctx.sync_currents(s.J, s.buff)
        s.ctx.filter_currents(s.J, s.buff, p.nfilter)
        return dict(J=s.J, sp=_particles(s, ("i_prev", "dx_prev")))
    if c["kind"] == "populate":
        for x in s.sp:
            x.npart = 0
        s.ctx.inject_uniform_maxwellians(s.sp[0], s.sp[1], s.inj)
        for x in s.sp:
            s.ctx.sort(x, abi.PIC_SORT_SPATIAL | abi.PIC_SORT_TILED | abi.PIC_SORT_SKIP_PREV)
        return dict(sp=_particles(s, ("w", "tag")), n=[x.npart for x in s.sp])
    if c["kind"] == "output":
        g = s.g
        s.mom.zero_()
        s.ctx.output_moment(s.sp, _moment(c, g, abi.PIC_MOM_N), s.mom, 0)
        s.ctx.output_moment(s.sp, _moment(c, g, abi.PIC_MOM_T, 0, 0), s.mom, 1)
        s.ctx.sync_moments(s.mom, 0, 2)
        s.ctx.output_field(s.EB, 1, 0, 3, abi.PIC_OUT_INTERP_EDGES | abi.PIC_OUT_TO_HAT, g.dx, (1, 1, 1), s.out)
        s.ctx.output_particles(s.sp[0], 10, g.dx, (0.0, 0.0, 0.0), s.rec[:3], s.rec[3:6], s.rec[6])
        return dict(mom=s.mom[:2], E=s.out, rec=s.rec)
    if c["kind"] == "wald":
        s.ctx.grpic_step(s.sp, s.fields, s.prm, island=s.island, step=s.k, match=s.ctx.match)
        s.k += 1
        return dict(fields=s.fields[:5], sp=_particles(s, ("tag",)))
    loss = s.ctx.gradient(s.sp, s.adj, s.EB, s.J, s.buff, s.prm, c["steps"], c["every"], s.lam)
    return dict(loss=loss, lam=s.lam, adj=[dict(lx=a.lx, lu=a.lu, lw=a.lw) for a in s.adj])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = case
    rb = 4 if c["real"] == "f32" else 8
    if c["kind"] == "wald":
        # cells of r < 6 on the log-spaced grid hold the pairs
        rh = 1.0 + math.sqrt(1.0 - c["a"] ** 2)
        frac = math.log(6.0 / (0.9 * rh)) / math.log(50.0 / (0.9 * rh))
        n = 2 * c["ppc"] * c["n1"] * c["n2"] * frac
        cells = c["n1"] * c["n2"]
        # i, dx, u, tag read, i, dx, u, the previous position and phi's momentum written; D, B and their copies
        # half a step back and J updated; ten implicit iterations and the metric
        return dict(bytes=n * (2 * 8 + 3 * rb + 2 + 2 * 16 + 3 * rb + rb) + cells * 2 * (12 + 6) * rb,
                    flops=n * 6000 + cells * 600)
    D, O = c["dim"], c["order"]
    cells = c["n1"] * c["n2"] * c["n3"]
    n = 2 * c["ppc"] * cells
    st = 8 * D + 4 * rb  # i, dx, u, w
    taps = (O + 1) ** D
    push = 6 * 2 * taps + 150 + D * 12 * (O + 1)
    dep = 3 * taps * 4 + D * 12 * (O + 1)
    if c["kind"] == "step":
        # state read and written (not w), tag read; E and B read and written, J written
        return dict(bytes=n * (2 * st - rb + 2) + cells * 15 * rb,
                    flops=n * (push + dep) + cells * (60 + 3 * 2 * 3 ** D * c["nfilter"]))
    if c["kind"] == "phases":
        # push: state read and written, previous position written; deposit: state and previous position read
        return dict(bytes=n * (2 * st - rb + 2 + 8 * D) + cells * 9 * rb,
                    flops=n * (push + dep) + cells * 3 * 2 * 3 ** D * c["nfilter"])
    if c["kind"] == "populate":
        return dict(bytes=n * (st + 2), flops=n * 200)
    if c["kind"] == "output":
        t = (2 * ((c["mom_order"] + 1) // 2) + 1) ** D
        return dict(bytes=n * (st + 2) + cells * 8 * rb + n // 20 * 7 * rb, flops=n * (2 * 2 * t + 40))
    K, every = c["steps"], c["every"]
    # forward steps, their recomputation (all segments but the last) and the reverse steps, which read a state
    # and update its gradients
    fwd = K + max(0, K - every)
    return dict(bytes=fwd * n * (2 * st - rb + 2) + K * n * (st + 2 + 2 * (D + 4) * rb) + (fwd + K) * cells * 15 * rb,
                flops=(fwd + 3 * K) * n * (push + dep))


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _spline(O, x):
    """Cardinal B-spline of order O at distance x."""
    x = x.abs()
    if O == 0:
        return torch.ones_like(x)
    if O == 1:
        return (1 - x).clamp_min(0)
    if O == 2:
        return torch.where(x < 0.5, 0.75 - x * x, 0.5 * (1.5 - x).clamp_min(0) ** 2)
    return torch.where(x < 1, 2 / 3 - x * x + 0.5 * x ** 3, (2 - x).clamp_min(0) ** 3 / 6)


def _first(O, x):
    """First node of the order-O support around x."""
    return torch.floor(x) - (O - 1) // 2 if O % 2 else torch.floor(x + 0.5) - 1


STAG = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (1, 1, 0)]


class Ref:
    """The periodic special-relativistic step on active cells, x1 fastest."""

    def __init__(self, g, prm):
        self.g, self.D, self.O, self.n, self.p = g, g.dim, g.order, g.n[:g.dim], prm
        self.third = 0.333333 if g.real == torch.float32 else 1.0 / 3.0  # the reference's single-precision constant

    def active(self, F):
        g, ng = self.g, self.g.ng
        z = slice(ng, -ng) if g.dim == 3 else slice(None)
        return F[:, z, ng:-ng, ng:-ng].double()

    def whole(self, A):
        ng = self.g.ng
        for d in (1, 2, 3)[(0 if self.D == 3 else 1):]:
            n = A.shape[d]
            A = torch.cat([A.narrow(d, n - ng, ng), A, A.narrow(d, 0, ng)], d)
        return A

    def flat(self, nodes):
        """Flat index of per-axis integer nodes, periodic."""
        f = 0
        for d in reversed(range(self.D)):
            f = f * self.n[d] + torch.remainder(nodes[d], self.n[d])
        return f

    def sh(self, A, d, k):  # A at cell index + k along axis d
        return torch.roll(A, -k, A.dim() - 1 - d)

    def faraday(self, E, B, frac):
        p, D = self.p, self.D
        dT = frac * p.correction * p.dt
        c1, c2 = (dT / p.dx ** 2, dT) if D == 2 else (dT / p.dx, dT / p.dx)
        d = lambda A, a: self.sh(A, a, 1) - A if a < D else 0.0
        return torch.stack([B[0] + c1 * (d(E[1], 2) - d(E[2], 1)), B[1] + c1 * (d(E[2], 0) - d(E[0], 2)),
                            B[2] + c2 * (d(E[0], 1) - d(E[1], 0))])

    def ampere(self, E, B, J):
        p, D = self.p, self.D
        dT = p.correction * p.dt
        c1, c2 = (dT / p.dx ** 2, dT) if D == 2 else (dT / p.dx, dT / p.dx)
        d = lambda A, a: A - self.sh(A, a, -1) if a < D else 0.0
        curl = [c1 * (d(B[2], 1) - d(B[1], 2)), c1 * (d(B[0], 2) - d(B[2], 0)), c2 * (d(B[1], 0) - d(B[0], 1))]
        return E + torch.stack(curl) - p.dt * p.q0 / (p.B0 * p.V0) * J

    def filter(self, J):
        for _ in range(self.p.nfilter):
            if self.D == 2:
                for a in range(2):
                    J = 0.25 * self.sh(J, a, -1) + 0.5 * J + 0.25 * self.sh(J, a, 1)
            else:
                # the reference's 3D stencil: its 1/32 group holds the x3 neighbours a second time in the
                # place of the last x2-x3 edge pair
                yz = self.sh(self.sh(J, 1, -1), 2, 1) + self.sh(self.sh(J, 1, 1), 2, -1)
                more = (self.sh(J, 2, -1) + self.sh(J, 2, 1) - yz) / 32
                for a in range(3):
                    J = 0.25 * self.sh(J, a, -1) + 0.5 * J + 0.25 * self.sh(J, a, 1)
                J = J + more
        return J

    def interp(self, F, x):
        D, O = self.D, self.O
        first, S = {}, {}
        for d in range(D):
            for s in (0, 1):
                y = x[d] - 0.5 * s
                first[d, s] = _first(O, y.detach())
                S[d, s] = [_spline(O, y - (first[d, s] + k)) for k in range(O + 1)]
        out = []
        for comp in range(6):
            A, v = F[comp].reshape(-1), 0.0
            st = STAG[comp]
            for t in range((O + 1) ** D):
                k = [t // (O + 1) ** d % (O + 1) for d in range(D)]
                w = 1.0
                for d in range(D):
                    w = w * S[d, st[d]][k[d]]
                v = v + w * A[self.flat([(first[d, st[d]] + k[d]).long() for d in range(D)])]
            out.append(v)
        return out

    def push(self, x, u, F, ndth):
        """New positions (unwrapped) and momenta."""
        D, p = self.D, self.p
        f = [v * p.dx if comp % 3 < D else v for comp, v in enumerate(self.interp(F, x))]
        e, b = [ndth * v for v in f[:3]], f[3:]
        cr = lambda a, c: [a[1] * c[2] - a[2] * c[1], a[2] * c[0] - a[0] * c[2], a[0] * c[1] - a[1] * c[0]]
        um = [a + c for a, c in zip(u, e)]
        k = ndth / torch.sqrt(1 + um[0] ** 2 + um[1] ** 2 + um[2] ** 2)
        t = [k * v for v in b]
        f2 = 2 / (1 + t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
        w = [(a + c) * f2 for a, c in zip(um, cr(um, t))]
        u1 = [a + c + d for a, c, d in zip(um, cr(w, t), e)]
        ig = 1 / torch.sqrt(1 + u1[0] ** 2 + u1[1] ** 2 + u1[2] ** 2)
        return [x[d] + u1[d] / p.dx * p.dt * ig for d in range(D)], u1

    def deposit(self, J, x0, x1, u, q):
        """J (3, cells flat) plus the current of charges q moving from x0 to x1."""
        D, O, N, p = self.D, self.O, self.O + 2, self.p
        base, iS, fS = [], [], []
        for d in range(D):
            b = torch.minimum(_first(O, x0[d].detach()), _first(O, x1[d].detach()))
            base.append(b)
            iS.append([_spline(O, x0[d] - (b + k)) for k in range(N)])
            fS.append([_spline(O, x1[d] - (b + k)) for k in range(N)])
        node = lambda ks: self.flat([(base[d] + ks[d]).long() for d in range(D)])
        Q = q / p.dt
        out = [J[0], J[1], J[2]]
        add = lambda comp, ks, v: out.__setitem__(comp, out[comp].index_add(0, node(ks), v))
        if D == 2:
            vz = q * u[2] / torch.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
            for j in range(N):
                acc = 0.0
                for i in range(N - 1):
                    acc = acc - Q * 0.5 * (fS[0][i] - iS[0][i]) * (fS[1][j] + iS[1][j])
                    add(0, (i, j), acc)
            for i in range(N):
                acc = 0.0
                for j in range(N - 1):
                    acc = acc - Q * 0.5 * (fS[0][i] + iS[0][i]) * (fS[1][j] - iS[1][j])
                    add(1, (i, j), acc)
                for j in range(N):
                    add(2, (i, j), vz * self.third * (fS[1][j] * (0.5 * iS[0][i] + fS[0][i]) +
                                                      iS[1][j] * (0.5 * fS[0][i] + iS[0][i])))
        else:
            for a in range(3):
                b, c = [d for d in range(3) if d != a]
                for j in range(N):
                    for k in range(N):
                        P = (iS[b][j] * iS[c][k] + fS[b][j] * fS[c][k] +
                             0.5 * (iS[c][k] * fS[b][j] + iS[b][j] * fS[c][k]))
                        acc = 0.0
                        for i in range(N - 1):
                            acc = acc - Q * self.third * (fS[a][i] - iS[a][i]) * P
                            ks = [0, 0, 0]
                            ks[a], ks[b], ks[c] = i, j, k
                            add(a, ks, acc)
        return torch.stack(out)


CHUNK = 1 << 22


def _shape3(r):
    n = tuple(reversed(r.n))
    return n if r.D == 3 else (1,) + n


def _ref_particles(r, sp, F, J):
    """Push and deposit of one species, in chunks: (dx, u) outputs and the new J."""
    p, D = r.p, r.D
    ndth = 0.5 * (sp.charge / sp.mass) * p.omegaB0 * p.dt
    dxs, us = [[] for _ in range(D)], [[] for _ in range(3)]
    for lo in range(0, sp.npart, CHUNK):
        sl = slice(lo, min(sp.npart, lo + CHUNK))
        x0 = [sp.i[d][sl].double() + sp.dx[d][sl].double() for d in range(D)]
        x1, u1 = r.push(x0, [v[sl].double() for v in sp.u], F, ndth)
        J = r.deposit(J, x0, x1, u1, sp.w[sl].double() * sp.charge)
        for d in range(D):
            dxs[d].append(x1[d] - torch.floor(x1[d]))
        for k in range(3):
            us[k].append(u1[k])
    return [torch.cat(v) for v in dxs], [torch.cat(v) for v in us], J


def exact(case, seed):
    c = case
    n = 2 * c["ppc"] * c["n1"] * c["n2"] * c.get("n3", 1)
    if c["kind"] in ("wald", "populate"):
        return None  # the metric's iterations and the random stream have no short restatement
    # larger boxes would take minutes of fp64 gathers and scatters
    if n * (c["order"] + 2) ** c["dim"] * (c["steps"] * 3 if c["kind"] == "gradient" else 1) > 9e9:
        return None
    s = prepare(c, seed)
    g, sp = s.g, s.sp
    r = Ref(g, s.prm)
    D, cells = r.D, c["n1"] * c["n2"] * c["n3"]
    F = r.active(s.EB)
    if c["kind"] == "output":
        return _exact_output(c, s, r)
    if c["kind"] == "gradient":
        return _exact_gradient(c, s, r)
    J = torch.zeros(3, cells, dtype=torch.float64, device="cuda")
    step = c["kind"] == "step"
    E, B = F[:3], F[3:]
    if step:
        B = r.faraday(E, B, 0.5)
    got = []
    for x in sp:
        prev = [v.double() for v in x.dx[:D]]
        dx, u, J = _ref_particles(r, x, torch.cat([E, B]), J)
        d = dict(i=[None] * D, dx=dx, u=u)
        if not step:
            d.update(i_prev=[None] * 3, dx_prev=prev)
        got.append(d)
    J = r.filter(J.reshape(3, *_shape3(r)))
    if not step:
        return dict(J=r.whole(J), sp=got)
    B = r.faraday(E, B, 0.5)
    E = r.ampere(E, B, J)
    return dict(EB=r.whole(torch.cat([E, B])), J=r.whole(J / s.prm.ppc0), sp=got)


def _exact_output(c, s, r):
    g, ng, O = s.g, s.g.ng, c["mom_order"]
    W = (O + 1) // 2
    cells = c["n1"] * c["n2"] * c["n3"]
    mom = torch.zeros(2, cells, dtype=torch.float64, device="cuda")
    for x in s.sp:
        cell = [i.long() for i in x.i]
        u0 = torch.sqrt(1 + sum(v.double() ** 2 for v in x.u))
        w = x.w.double() / (2.0 * c["ppc"]) / g.dx ** 3
        S = [[_spline(O, x.dx[d].double() - (q - W + 0.5)) for q in range(2 * W + 1)] for d in range(3)]
        for t in range((2 * W + 1) ** 3):
            k = [t // (2 * W + 1) ** d % (2 * W + 1) for d in range(3)]
            at = r.flat([cell[d] + k[d] - W for d in range(3)])
            v = w * S[0][k[0]] * S[1][k[1]] * S[2][k[2]]
            mom[0].index_add_(0, at, v)
            mom[1].index_add_(0, at, v * x.mass * u0)
    full = torch.zeros((2,) + tuple(s.mom.shape[1:]), dtype=torch.float64, device="cuda")
    full[:, ng:-ng, ng:-ng, ng:-ng] = mom.reshape(2, *_shape3(r))
    F = r.active(s.EB)[:3]
    E = torch.stack([sum(r.sh(r.sh(F[a], b, i), d, j) for i in (0, 1) for j in (0, 1)) * 0.25 * g.dx
                     for a, b, d in ((0, 1, 2), (1, 0, 2), (2, 0, 1))])
    x, m = s.sp[0], s.sp[0].npart // 10 * 10
    rec = [((x.i[d].double() + x.dx[d].double()) * g.dx)[:m:10] for d in range(3)]
    rec += [v.double()[:m:10] for v in x.u] + [x.w.double()[:m:10]]
    return dict(mom=full, E=E, rec=rec)


def _exact_gradient(c, s, r):
    from torch.utils.checkpoint import checkpoint
    g, p, D, nsp = s.g, r.p, r.D, len(s.sp)
    X = [[(x.i[d].double() + x.dx[d].double()).requires_grad_() for d in range(D)] for x in s.sp]
    U = [[v.double().requires_grad_() for v in x.u] for x in s.sp]
    Wt = [x.w.double().requires_grad_() for x in s.sp]
    F0 = r.active(s.EB).requires_grad_()
    cells = c["n1"] * c["n2"]

    def step(F, *state):
        E, B = F[:3], r.faraday(F[:3], F[3:], 0.5)
        J = torch.zeros(3, cells, dtype=torch.float64, device="cuda")
        new = []
        for k in range(nsp):
            x, u, w = state[k * (D + 4):k * (D + 4) + D], state[k * (D + 4) + D:k * (D + 4) + D + 3], state[k * (D + 4) + D + 3]
            ndth = 0.5 * (s.sp[k].charge / s.sp[k].mass) * p.omegaB0 * p.dt
            x1, u1 = r.push(list(x), list(u), torch.cat([E, B]), ndth)
            J = r.deposit(J, x, x1, u1, w * s.sp[k].charge)
            new += [*x1, *u1, w]
        J = r.filter(J.reshape(3, *_shape3(r)))
        B = r.faraday(E, B, 0.5)
        return (torch.cat([r.ampere(E, B, J), B]), *new)

    with torch.enable_grad():
        F, state = F0, [t for k in range(nsp) for t in (*X[k], *U[k], Wt[k])]
        for _ in range(c["steps"]):
            F, *state = checkpoint(step, F, *state, use_reentrant=False)
        E = F[:3]
        h = g.dx * g.dx
        loss = ((E[0] ** 2 + E[1] ** 2) * h + E[2] ** 2).sum() * h
        loss.backward()
    lam = torch.zeros(s.lam.shape, dtype=torch.float64, device="cuda")
    ng = g.ng
    lam[:, :, ng:-ng, ng:-ng] = F0.grad
    return dict(loss=float(loss.detach()), lam=lam,
                adj=[dict(lx=[x.grad for x in X[k]], lu=[u.grad for u in U[k]], lw=Wt[k].grad) for k in range(nsp)])
