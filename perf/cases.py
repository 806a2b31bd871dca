"""Timed cases: what users of the framework run, through its public entry points.

Kinds of case and what each stands for:

  request  a step plan (plan.StepPlan: one CUDA graph per time step) that is
           given a new state, as a server or a parameter study does with every
           request, and advances it ``steps`` steps.  Precision form, box and
           SFS closure are options of the plan.
  batch    a batch plan (plan.BatchPlan): the active requests of the
           continuous-batching server, of uneven sizes, advanced together.
  pyflow   the drop-in PyFlow.run path: host-driven Domain.forwardStep calls
           (ops.forward_step), FP64, the reference's BiCGStab.
  window   a differentiable LES window (adjoint.forward_step with 'tensor' SFS
           stresses, loss against filtered targets): forward and backward.
  slab     the x-slab decomposition (slab.SlabDomain) with its distributed
           BiCGStab, the slabs held by one process.
  mlp      the tensor-core MLP SGS closure alone, as an LES step calls it.
  source   the reference's gated 'source' ML closure alone, as every RK stage
           of an LES with that closure calls it.

Velocity fields are the decaying-turbulence fields of the framework
(spectrum k^4 exp(-2 (k/k0)^2), urms = 1, seeded).  A pass that advances a
state loads it first, so every pass does the same work.  Velocities come out
as they are held (FP64).  The mixed forms compute their fluxes in FP32, which
leaves the accumulated pressure with an FP32 error (1e-7 to 1e-6 of its norm
against 64 bits): as a program that writes snapshots does, the pressure of
those forms is taken out in FP32, that of the FP64 forms in FP64.
"""
import math

import numpy as np
import torch

import pyflow_b200.adjoint as adjoint
import pyflow_b200.initial as initial
import pyflow_b200.ops as ops
import pyflow_b200.sfsmodel_ML as sfs_ml
import pyflow_b200.sfsmodel_mlp as sfs_mlp
from pyflow_b200.plan import BatchPlan, Member, StepPlan
from pyflow_b200.slab import LocalSlabs, SlabDomain

DEV = "cuda"
RHO = 1.0
TOL = 1e-10       # the reference configurations' pressure tolerance
MAX_IT = 20000
CS = 0.18         # Smagorinsky constant

STEP_KINDS = ("request", "pyflow", "window", "slab")


def _box(kind, nx, ny, nz, **more):
    """A case on an nx x ny x nz grid of the [0, 2 pi]^3 box: viscosity and
    time step as in the serving stream (nu = 0.02 * 32 / n, CFL 0.3)."""
    n = max(nx, ny, nz)
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "k0": 4.0,
         "nu": 0.02 * 32 / n, "dt": 0.3 * (2 * math.pi / n) / 4.0}
    c.update(more)
    return c


def listed():
    return [
        # the smallest serving request: latency and launches are all there is
        _box("request", 32, 32, 32, name="request_32", prec="mixed_mg", closure="none", steps=10),
        # plain FP64 DNS, the reference's own algorithm on its own test size
        _box("request", 64, 64, 64, name="request_64_fp64", prec="fp64", closure="none", steps=2,
             nu=0.01, dt=0.005),
        # decaying turbulence DNS, the accuracy workload
        _box("request", 128, 128, 128, name="request_128", prec="mixed_mg", closure="none",
             steps=5, nu=0.005, dt=0.0025),
        # the large single-box DNS, the headline workload
        _box("request", 512, 512, 512, name="request_512", prec="mixed_mg", closure="none",
             steps=2, k0=8.0, nu=0.0012, dt=0.001),
        # a box of uneven, partly odd extents: nothing halves or divides evenly
        _box("request", 90, 77, 63, name="request_90x77x63", prec="mixed_mg", closure="none",
             steps=3),
        # LES at the training size with the eddy-viscosity closure in the graph
        _box("request", 64, 64, 64, name="les_64", prec="mixed_mg", closure="smagorinsky",
             steps=5, nu=0.001, dt=0.005),
        # the server's active set: eight requests of the stream's sizes
        {"name": "batch_8", "kind": "batch", "sizes": "32,48,64,64,96,96,128,192", "steps": 4},
        # PyFlow.run's step, host-driven
        _box("pyflow", 96, 96, 96, name="pyflow_96", steps=1, nu=0.005, dt=0.0025),
        # a-posteriori training: two differentiable LES steps and their adjoint
        _box("window", 64, 64, 64, name="window_64", steps=2, nu=0.001, dt=0.005),
        # two slabs of a box that would be split over ranks
        _box("slab", 96, 64, 64, name="slab_96x64x64", slabs=2, steps=1),
        # the MLP closure at the DNS accuracy size
        {"name": "mlp_128", "kind": "mlp", "nx": 128, "ny": 128, "nz": 128, "k0": 4.0},
        # the source closure at the LES training size
        {"name": "source_64", "kind": "source", "nx": 64, "ny": 64, "nz": 64, "k0": 4.0},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["request", "request", "request", "request", "batch", "pyflow", "window",
                       "slab", "mlp", "source"])
    if kind == "request":
        what = rng.choice(["even", "even", "any", "fp64", "les"])
        if what == "even":       # boxes that users choose: multiples of 16
            n = [16 * _size(rng, 2, 24) for _ in range(3)]
            return _box("request", *n, prec="mixed_mg", closure="none", steps=rng.randint(1, 3),
                        k0=rng.choice([4.0, 6.0]))
        if what == "any":        # odd and ragged ones
            n = [_size(rng, 17, 110) for _ in range(3)]
            return _box("request", *n, prec=rng.choice(["mixed", "mixed_mg"]), closure="none",
                        steps=rng.randint(1, 3))
        if what == "fp64":
            n = [_size(rng, 20, 110) for _ in range(3)]
            return _box("request", *n, prec="fp64", closure="none", steps=1)
        n = [4 * _size(rng, 6, 32) for _ in range(3)]
        return _box("request", *n, prec=rng.choice(["mixed_mg", "fp64"]),
                    closure=rng.choice(["smagorinsky", "gradient"]), steps=rng.randint(1, 3),
                    nu=0.002)
    if kind == "batch":
        sizes = [rng.choice([32, 40, 48, 64, 80, 96, 128, 160, 192])
                 for _ in range(rng.randint(2, 8))]
        return {"kind": "batch", "sizes": ",".join(str(n) for n in sizes),
                "steps": rng.randint(1, 4)}
    if kind in ("pyflow", "window"):
        n = [_size(rng, 20, 96) for _ in range(3)]
        return _box(kind, *n, steps=rng.randint(1, 2))
    if kind == "slab":
        return _box("slab", _size(rng, 24, 96), _size(rng, 20, 80), _size(rng, 20, 80),
                    slabs=rng.randint(1, 3), steps=1)
    hi = 256 if kind == "mlp" else 96
    return {"kind": kind, "nx": _size(rng, 16, hi), "ny": _size(rng, 16, hi),
            "nz": _size(rng, 16, hi), "k0": 4.0}


# ---------------------------------------------------------------- inputs
def _shape(c):
    return (int(c["nx"]), int(c["ny"]), int(c["nz"]))


def _spacing(shape):
    return tuple(2 * math.pi / n for n in shape)


def _field(shape, k0, seed):
    return [t.contiguous() for t in initial.spectral_velocity_device(
        shape, k0=k0, seed=seed, device=DEV, noise="device")]


def _sizes(c):
    return [int(x) for x in c["sizes"].split(",")]


def _seed(seed, i=0):
    return int(seed) * 64 + i


def _request_field(c, seed):
    return _field(_shape(c), c["k0"], _seed(seed))


def _batch_fields(c, seed):
    return [_field((n, n, n), 4.0, _seed(seed, i)) for i, n in enumerate(_sizes(c))]


def _window_inputs(c, seed):
    """Initial velocity, targets after every step (between the initial field
    and another one, both discretely divergence free) and six SFS stresses of
    a gradient model's size."""
    shape, sp = _shape(c), _spacing(_shape(c))
    u0 = _request_field(c, seed)
    other = _field(shape, c["k0"], _seed(seed, 1))
    targets = [[0.98 * a + 0.02 * b for a, b in zip(u0, other)] for _ in range(c["steps"])]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(_seed(seed, 2))
    scale = sp[0] ** 2 / 12.0 * c["k0"] ** 2
    sfs = [scale * torch.randn((6,) + shape, generator=gen, dtype=torch.float64, device=DEV)
           for _ in range(c["steps"])]
    return u0, targets, sfs


def _source_weights(seed):
    """The closure network as created from a seed (CPU generator, so that the
    oracle makes the same one)."""
    state = torch.random.get_rng_state()
    torch.manual_seed(int(seed) % (1 << 31))
    net = sfs_ml.GatedClosureNet()
    torch.random.set_rng_state(state)
    return net


def _coef(c, closure):
    h = _spacing(_shape(c))[0]
    return RHO * (CS * h) ** 2 if closure == "smagorinsky" else h * h / 12.0


class _Obj:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        start = _batch_fields(c, seed)
        members = []
        for n, f0 in zip(_sizes(c), start):
            f = [t.clone() for t in f0] + [torch.zeros_like(f0[0]) for _ in range(2)]
            members.append(Member(*f, _spacing((n, n, n)), 0.02 * 32 / n, RHO,
                                  0.3 * (2 * math.pi / n) / 4.0, min_res=TOL, max_it=MAX_IT,
                                  prec="mixed_mg"))
        return _Obj(kind=kind, start=start, members=members, plan=BatchPlan(members),
                    steps=c["steps"])
    shape = _shape(c)
    sp = _spacing(shape)
    if kind == "request":
        u0 = _request_field(c, seed)
        f = [t.clone() for t in u0] + [torch.zeros_like(u0[0]) for _ in range(2)]
        more = {}
        if c["closure"] != "none":
            more = {"closure": c["closure"], "coef": _coef(c, c["closure"])}
        plan = StepPlan(*f, sp, c["nu"], RHO, c["dt"], min_res=TOL, max_it=MAX_IT,
                        prec=c["prec"], **more)
        return _Obj(kind=kind, start=u0, fields=f, plan=plan, steps=c["steps"], prec=c["prec"])
    if kind == "pyflow":
        u0 = _request_field(c, seed)
        f = [t.clone() for t in u0] + [torch.zeros_like(u0[0]) for _ in range(2)]
        return _Obj(kind=kind, start=u0, fields=f, case=c, sp=sp)
    if kind == "window":
        u0, targets, sfs = _window_inputs(c, seed)
        return _Obj(kind=kind, start=u0, targets=targets, sfs=sfs, case=c, sp=sp)
    if kind == "slab":
        u0 = _request_field(c, seed)
        D = SlabDomain(shape, sp, c["nu"], RHO, c["dt"], LocalSlabs(c["slabs"]), min_res=TOL,
                       max_it=MAX_IT)
        return _Obj(kind=kind, start=u0, domain=D, steps=c["steps"])
    u = _field(shape, c["k0"], _seed(seed))
    if kind == "mlp":
        params = sfs_mlp.xavier_init(_seed(seed, 3))
        return _Obj(kind=kind, u=u, sp=sp, wpack=torch.as_tensor(sfs_mlp.pack(params)).to(DEV))
    net = _source_weights(_seed(seed, 4)).to(DEV)
    geo = _Obj(dx=sp[0], type="uniform")
    model = sfs_ml.residual_stress(_Obj(), _Obj(device=torch.device(DEV)), geo, model=net)
    return _Obj(kind=kind, u=u, model=model)


# ------------------------------------------------------------------- run
def _load(fields, start):
    for d, s in zip(fields, start):
        d.copy_(s)
    for d in fields[len(start):]:
        d.zero_()


def _mse(a, b):
    return sum(torch.mean((x - y) ** 2) for x, y in zip(a, b)) / 3.0


def _window(step, u0, targets, sfs):
    """Loss of the window, its final velocity and the gradients of the loss
    with respect to the initial velocity and the stresses."""
    leaves = [t.detach().requires_grad_(True) for t in list(u0) + list(sfs)]
    cur, loss = tuple(leaves[:3]), 0.0
    for n, tgt in enumerate(targets):
        cur = step(cur, leaves[3 + n])
        loss = loss + _mse(cur, tgt)
    grads = torch.autograd.grad(loss, leaves)
    return [t.detach() for t in cur], list(grads)


def _out(fields, prec):
    u, v, w, p = fields[:4]
    return {"u": u, "v": v, "w": w, "p": p if prec == "fp64" else p.float()}


def run(state):
    s = state
    if s.kind == "request":
        _load(s.fields, s.start)
        s.plan.launch(s.steps)
        return _out(s.fields, s.prec)
    if s.kind == "batch":
        for m, f0 in zip(s.members, s.start):
            _load(m.fields, f0)
        s.plan.launch(s.steps)
        return [_out(m.fields, m.prec) for m in s.members]
    if s.kind == "pyflow":
        c = s.case
        _load(s.fields, s.start)
        for _ in range(c["steps"]):
            ops.forward_step(*s.fields, s.sp, c["nu"], RHO, c["dt"], min_res=TOL, max_it=MAX_IT)
        return _out(s.fields, "fp64")
    if s.kind == "window":
        c = s.case

        def step(cur, F):
            return adjoint.forward_step(*cur, s.sp, c["nu"], RHO, c["dt"], sfs=F)
        vel, grads = _window(step, s.start, s.targets, s.sfs)
        return {"vel": vel, "grads": grads}
    if s.kind == "slab":
        s.domain.set_state(*s.start)
        for _ in range(s.steps):
            s.domain.forward_step()
        return {k: s.domain.gather(k) for k in "uvwp"}
    if s.kind == "mlp":
        out, _, _, _ = sfs_mlp.closure(*s.u, s.sp, s.wpack, s.sp[0])
        return {"stress": out}
    s.model.update(*s.u)
    m = s.model
    return {"G": [m.GX, m.GY, m.GZ], "S": list(m.face_sources())}


# ------------------------------------------------------------------ work
def work(case):
    """Bytes: the state (or closure input) read once and the result written
    once, FP64.  Flops: the stencils of the steps and one solve of the
    pressure equation by fast transforms, or the network's products."""
    c, kind = case, case["kind"]
    if kind == "batch":
        cells = [n ** 3 for n in _sizes(c)]
        return {"bytes": 64.0 * sum(cells),
                "flops": float(c["steps"] * sum(n * (600 + 10 * math.log2(n)) for n in cells))}
    n = float(np.prod([float(a) for a in _shape(c)]))
    step = n * (600 + 10 * math.log2(n))
    if kind == "mlp":
        return {"bytes": 72.0 * n, "flops": 2.0 * (9 * 128 + 128 * 128 + 128 * 6) * n}
    if kind == "source":
        return {"bytes": 72.0 * n, "flops": 2.0 * (3 * 273 * 200 + 2 * 200 * 200 + 200 * 18) * n}
    if kind == "window":
        # velocity in and out, its gradient, targets, stresses and theirs
        return {"bytes": 8.0 * n * (9 + c["steps"] * (3 + 12)), "flops": 3.0 * c["steps"] * step}
    extra = {"none": 0, "smagorinsky": 80, "gradient": 80}[c.get("closure", "none")]
    return {"bytes": 64.0 * n, "flops": c["steps"] * (step + extra * n)}


# ----------------------------------------------------------------- exact
def _at(a, i, j, k):
    """a at (i, j, k) cells away, periodic (last three dimensions)."""
    sh, dims = [], []
    for s, d in ((i, -3), (j, -2), (k, -1)):
        if s:
            sh.append(-s)
            dims.append(d)
    return torch.roll(a, sh, dims) if sh else a


E = ((1, 0, 0), (0, 1, 0), (0, 0, 1))


def _p(a, d):
    return _at(a, *E[d])


def _m(a, d):
    return _at(a, *(-x for x in E[d]))


def _edge(a, d, e):
    """Mean of the four cells around the edge below a cell."""
    b = _m(a, d)
    return 0.25 * (a + b + _m(a, e) + _m(b, e))


def _rhs(vel, sp, mu, rho, visc=None, sfs=None):
    """Staggered second-order right-hand side (convective and viscous
    fluxes, SFS stresses at cell centres)."""
    h = sp
    div3 = sum((_p(vel[d], d) - vel[d]) / h[d] for d in range(3)) / 3.0
    out = [0.0, 0.0, 0.0]
    for d in range(3):
        nu = (mu if visc is None else visc) / rho
        F = ((_p(vel[d], d) - vel[d]) / h[d] - div3) * (2.0 * nu)
        if sfs is not None:
            F = F + sfs[d]
        c = 0.5 * (_p(vel[d], d) + vel[d])
        F = F - c * c
        out[d] = out[d] + (F - _m(F, d)) / h[d]
    for n, (d, e) in enumerate(((0, 1), (0, 2), (1, 2))):
        nu = (mu if visc is None else _edge(visc, d, e)) / rho
        F = ((_p(vel[d], e) - vel[d]) / h[e] + (_p(vel[e], d) - vel[e]) / h[d]) * nu
        if sfs is not None:
            F = F + _edge(sfs[3 + n], d, e)
        C = 0.25 * (vel[d] + _m(vel[d], e)) * (vel[e] + _m(vel[e], d))
        out[d] = out[d] + (F - _m(F, e)) / h[e] - (_p(C, e) - C) / h[e]
        out[e] = out[e] + (F - _m(F, d)) / h[d] - (_p(C, d) - C) / h[d]
    return out


def _poisson(src, sp):
    """Zero-mean solution of the 7-point Laplacian, by Fourier transform."""
    lam = 0.0
    for d in range(3):
        n = src.shape[d]
        k = torch.arange(n // 2 + 1 if d == 2 else n, dtype=torch.float64, device=src.device)
        s = torch.sin(math.pi * k / n)
        shape = [1, 1, 1]
        shape[d] = -1
        lam = lam - (4.0 * s * s / sp[d] ** 2).reshape(shape)
    lam = torch.where(lam == 0, torch.ones_like(lam), lam)
    hat = torch.fft.rfftn(src) / lam
    mask = torch.ones_like(lam)
    mask[0, 0, 0] = 0.0
    return torch.fft.irfftn(hat * mask, s=src.shape)


def _grad9(vel, sp):
    """Cell-centred gradients [component][direction]."""
    out = []
    for c in range(3):
        row, mid = [], 0.5 * (_p(vel[c], c) + vel[c])
        for d in range(3):
            if d == c:
                row.append((_p(vel[c], c) - vel[c]) / sp[c])
            else:
                row.append((_p(mid, d) - _m(mid, d)) / (2.0 * sp[d]))
        out.append(row)
    return out


def _closure_fields(closure, vel, sp, nu, coef):
    if closure == "none":
        return None, None
    g = _grad9(vel, sp)
    if closure == "smagorinsky":
        tr = (g[0][0] + g[1][1] + g[2][2]) / 3.0
        ss = sum((g[d][d] - tr) ** 2 for d in range(3))
        for d, e in ((0, 1), (0, 2), (1, 2)):
            ss = ss + 2.0 * (0.5 * (g[d][e] + g[e][d])) ** 2
        return nu + coef * torch.sqrt(ss), None
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    return None, torch.stack([coef * sum(g[a][d] * g[b][d] for d in range(3)) for a, b in pairs])


def _exact_step(vel, sp, nu, dt, visc=None, sfs=None):
    """RK4 predictor (stage states u + dt/2 k, the last one too), projection.
    Returns the new velocity and the pressure increment."""
    k, ksum, cur = None, None, list(vel)
    for s in range(4):
        k = _rhs(cur, sp, nu, RHO, visc, sfs)
        wgt = (1.0, 2.0, 2.0, 1.0)[s]
        ksum = [wgt * a for a in k] if ksum is None else [b + wgt * a for a, b in zip(k, ksum)]
        cur = [a + 0.5 * dt * b for a, b in zip(vel, k)]
    out = [a + dt / 6.0 * b for a, b in zip(vel, ksum)]
    div = sum((_p(out[d], d) - out[d]) / sp[d] for d in range(3))
    DP = _poisson(div, sp) * (RHO / dt)
    return [out[d] - dt / RHO * (DP - _m(DP, d)) / sp[d] for d in range(3)], DP


def _exact_steps(vel, sp, nu, dt, steps, closure="none", coef=0.0):
    p = 0.0
    for _ in range(steps):
        visc, sfs = _closure_fields(closure, vel, sp, nu, coef)
        vel, DP = _exact_step(vel, sp, nu, dt, visc, sfs)
        p = p + DP
    return dict(zip("uvwp", list(vel) + [p]))


def _exact_mlp(vel, sp, params):
    g = torch.stack([a for row in _grad9(vel, sp) for a in row])
    g2 = torch.mean(g * g)
    x = g.reshape(9, -1) / torch.sqrt(g2)
    W = [torch.as_tensor(params[k], device=DEV) for k in ("W1", "W2", "W3")]
    b = [torch.as_tensor(params[k], dtype=torch.float64, device=DEV) for k in ("b1", "b2", "b3")]
    for n in range(3):
        x = W[n].to(torch.bfloat16).double() @ x + b[n][:, None]
        x = torch.tanh(x) if n < 2 else x
    return (x * (sp[0] ** 2 * g2)).reshape((6,) + tuple(vel[0].shape))


def _exact_source(vel, dx, net):
    """The gated network in FP64 on central-difference features."""
    norm = torch.tensor(sfs_ml.NORM, dtype=torch.float64, device=DEV)
    mid = [0.5 * (_p(vel[c], c) + vel[c]) for c in range(3)]
    first = [(_p(a, d) - _m(a, d)) / (2 * dx) for a in mid for d in range(3)]
    second = [(_p(a, d) - 2 * a + _m(a, d)) / (dx * dx) for a in mid for d in range(3)]
    F = torch.stack(mid + first + second) / norm[:, None, None, None]
    x = [F]
    for s in (1, 2):
        for d in range(3):
            x += [_at(F, *(s * e for e in E[d])), _at(F, *(-s * e for e in E[d]))]
    x = torch.cat(x).reshape(273, -1)
    P = {k: v.detach().to(DEV, torch.float64) for k, v in net.named_parameters()}

    def lin(nm, a):
        return P[nm + ".weight"] @ a + P[nm + ".bias"][:, None]
    h = torch.tanh(lin("fc2", torch.tanh(lin("fc1", x)))) * torch.tanh(lin("fcG", x))
    h = torch.tanh(lin("fc3", h)) * torch.tanh(lin("fcG2", x))
    o = lin("fc4", h).reshape((18,) + tuple(vel[0].shape))
    G = [sum((_p(o[3 * c + d], d) - _m(o[3 * c + d], d)) / (2 * dx) for d in range(3))
         for c in range(3)]
    return {"G": G, "S": [0.5 * (G[d] + _m(G[d], d)) for d in range(3)]}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        return [_exact_steps(f, _spacing((n, n, n)), 0.02 * 32 / n,
                             0.3 * (2 * math.pi / n) / 4.0, c["steps"])
                for n, f in zip(_sizes(c), _batch_fields(c, seed))]
    shape = _shape(c)
    sp = _spacing(shape)
    if kind == "window":
        u0, targets, sfs = _window_inputs(c, seed)

        def step(cur, F):
            return _exact_step(cur, sp, c["nu"], c["dt"], sfs=F)[0]
        vel, grads = _window(step, u0, targets, sfs)
        return {"vel": vel, "grads": grads}
    if kind in STEP_KINDS:
        closure = c.get("closure", "none")
        return _exact_steps(_request_field(c, seed), sp, c["nu"], c["dt"], c["steps"], closure,
                            _coef(c, closure))
    u = _field(shape, c["k0"], _seed(seed))
    if kind == "mlp":
        return {"stress": _exact_mlp(u, sp, sfs_mlp.xavier_init(_seed(seed, 3)))}
    return _exact_source(u, sp[0], _source_weights(_seed(seed, 4)))
