"""What is timed: right-hand sides, time steps and gradients of the suite's
operators through the public API, at the sizes users run.

A case is a dict of plain values.  ``kind`` names the call a program makes:

* ``rhs``       ``compiled = actx.compile(rhs); compiled(*args)``, the suite's hot loop;
* ``step``      one LSRK(5,4) step of a plan (five fused stages);
* ``rhs_vjp``   ``RHSFunction``: an RHS and the gradient of a product with it
                (forward and backward);
* ``gradient``  ``WaveMisfitFunction``: receiver traces of a few wave steps and
                their gradients (a whole forward and reverse sweep);
* ``ensemble``  a batch of Maxwell members on uneven meshes, autotuned within an
                error bound and replayed as a CUDA graph.

``n`` is the number of cells per axis of a box mesh: 6 n^3 tetrahedra or 2 n^2
triangles.  Inputs come from the seed alone: a seeded mix of smooth waves around
the benchmark's problem definitions.  ``exact`` evaluates the same operators in
plain torch in 64 bits: its own nodes, reference operators (in 50-digit
arithmetic), mesh and face matching.
"""

from __future__ import annotations

import itertools
import math
import random
from decimal import Decimal, localcontext
from functools import lru_cache

import numpy as np
import torch

BOX = {"wave": (-1.0, 1.0), "euler": (-0.5, 0.5), "maxwell": (0.0, 1.0)}
PARAMS = {"wave": (1.0,), "euler": (1.4,), "maxwell": (1.0, 1.0, 1.0)}
NFIELDS = {3: {"wave": 4, "euler": 5, "maxwell": 6},
           2: {"wave": 3, "euler": 4, "maxwell": 3}}
DEVICE = "cuda"

# {{{ the cases


def listed() -> list[dict]:
    def case(name, kind, equation, order, n, dim=3, precision="fp64", **kw):
        return dict(name=name, kind=kind, equation=equation, order=order, n=n,
                    dim=dim, precision=precision, **kw)

    return [
        # the suite's CI and debugging size (tiny_: 1e3 DOFs per field): a call
        # whose time is launches and latency
        case("wave-p2-tiny", "rhs", "wave", 2, 6),
        # a run on triangles (the suite's --dims 2)
        case("euler-p3-2d", "rhs", "euler", 3, 200, dim=2),
        # the benchmark sweep's largest element count (large_: 2e7 DOFs per field)
        case("wave-p1-large", "rhs", "wave", 1, 95),
        # the suite's default budget (4e6 DOFs per field), odd element count per axis
        case("wave-p3", "rhs", "wave", 3, 33),
        # time stepping at the default budget
        case("euler-p2-step", "step", "euler", 2, 41),
        # the default budget at the highest order
        case("euler-p4", "rhs", "euler", 4, 27),
        # the benchmark sweep's dominant case
        case("maxwell-p4-large", "rhs", "maxwell", 4, 46),
        # FP32 arithmetic on FP64 states: one large RHS, and time stepping
        case("maxwell-p3-mixed-large", "rhs", "maxwell", 3, 56, precision="fp32-mixed"),
        case("euler-p3-mixed-step", "step", "euler", 3, 32, precision="fp32-mixed"),
        # many uneven members in one launch
        case("maxwell-p3-ensemble", "ensemble", "maxwell", 3, 26, precision="fp32-mixed",
             members=16),
        # an RHS with its backward pass inside a user's autograd program
        case("euler-p3-vjp", "rhs_vjp", "euler", 3, 24),
        # a full-waveform gradient: forward and reverse sweep
        case("wave-p3-gradient", "gradient", "wave", 3, 14, steps=3),
    ]


def draw(rng: random.Random) -> dict:
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rhs"] * 7 + ["step"] * 2 + ["rhs_vjp", "gradient", "ensemble"])
    order = rng.randint(1, 4)
    top = {1: 95, 2: 70, 3: 56, 4: 46}[order]
    if kind == "rhs":
        eq = rng.choice(["wave", "euler", "maxwell"])
        if rng.random() < 0.25:
            return dict(kind=kind, equation=eq, order=order, n=size(5, 300), dim=2,
                        precision="fp64")
        return dict(kind=kind, equation=eq, order=order, n=size(3, top), dim=3,
                    precision=rng.choice(["fp64", "fp64", "fp32-mixed"]))
    if kind == "step":
        return dict(kind=kind, equation=rng.choice(["wave", "euler", "maxwell"]),
                    order=order, n=size(4, top // 2), dim=3,
                    precision=rng.choice(["fp64", "fp32-mixed"]))
    if kind == "rhs_vjp":
        return dict(kind=kind, equation=rng.choice(["wave", "euler"]), order=order,
                    n=size(4, top // 2), dim=3, precision="fp64")
    if kind == "gradient":
        return dict(kind=kind, equation="wave", order=order, n=size(4, top // 4), dim=3,
                    precision="fp64", steps=rng.randint(2, 4))
    return dict(kind=kind, equation="maxwell", order=order, n=size(8, top // 2), dim=3,
                precision="fp32-mixed", members=rng.randint(3, 17))


def _member_sizes(case: dict) -> list[int]:
    """Cells per axis of each ensemble member, n/2 .. n (uneven)."""
    rng = random.Random(1000 * case["n"] + case["members"])
    return [rng.randint(max(2, case["n"] // 2), case["n"]) for _ in range(case["members"])]


# }}}

# {{{ plain reference element (50 digits) and box mesh, shared by the inputs and exact()


def _gll01(n: int) -> list[Decimal]:
    """Gauss-Lobatto-Legendre points of degree n <= 4 on [0, 1]."""
    half = Decimal(1) / 2
    inner = {1: [], 2: [Decimal(0)], 3: [Decimal(1) / Decimal(5).sqrt()],
             4: [Decimal(0), (Decimal(3) / Decimal(7)).sqrt()]}[n]
    x = sorted({s * v for v in inner for s in (1, -1)} | {Decimal(1), Decimal(-1)})
    return [half * (v + 1) for v in x]


def _recursive_node(alpha: tuple) -> list[Decimal]:
    """Barycentric coordinates of a node of the recursive interpolation family
    (Isaac, SIAM J. Sci. Comput. 42, 2020) on Gauss-Lobatto-Legendre points."""
    n = sum(alpha)
    g = _gll01(n) if n > 0 else [Decimal(1)]
    if len(alpha) == 2:
        return [g[alpha[0]], g[alpha[1]]]
    b, wsum = [Decimal(0)] * len(alpha), Decimal(0)
    for i in range(len(alpha)):
        w = g[n - alpha[i]]
        if w == 0:
            continue
        sub = _recursive_node(alpha[:i] + alpha[i + 1:])
        for k, v in zip([k for k in range(len(alpha)) if k != i], sub):
            b[k] += w * v
        wsum += w
    return [v / wsum for v in b]


def _matmul(a, b):
    bt = list(zip(*b))
    return [[sum((x * y for x, y in zip(r, c) if x and y), Decimal(0)) for c in bt] for r in a]


def _inverse(a):
    n = len(a)
    m = [list(r) + [Decimal(int(i == k)) for k in range(n)] for i, r in enumerate(a)]
    for c in range(n):
        p = max(range(c, n), key=lambda r: abs(m[r][c]))
        m[c], m[p] = m[p], m[c]
        piv = m[c][c]
        m[c] = [v / piv for v in m[c]]
        for r in range(n):
            if r != c and m[r][c]:
                f = m[r][c]
                m[r] = [v - f * w for v, w in zip(m[r], m[c])]
    return [r[n:] for r in m]


def _exponents(dim: int, order: int) -> list[tuple]:
    if dim == 0:
        return [()]
    return [rest + (last,) for last in range(order + 1)
            for rest in _exponents(dim - 1, order - last)]


def _monomial_mass(exps, dim):
    """Integrals of x^(a+b) over the unit simplex."""
    def integral(a):
        return (Decimal(math.prod(math.factorial(k) for k in a))
                / Decimal(math.factorial(sum(a) + dim)))
    return [[integral(tuple(p + q for p, q in zip(a, b))) for b in exps] for a in exps]


@lru_cache(maxsize=None)
def _element(dim: int, order: int) -> dict:
    """Nodes and operators on the unit simplex: strong and weak derivatives and,
    per face f (opposite vertex f), its nodes and LIFT columns."""
    with localcontext() as ctx:
        ctx.prec = 50
        exps = _exponents(dim, order)
        alphas = [(order - sum(a),) + a for a in exps]
        bary = [_recursive_node(a) for a in alphas]

        def vandermonde(points, es):
            return [[math.prod((x**k for x, k in zip(p, a) if k), start=Decimal(1))
                     for a in es] for p in points]

        v = vandermonde([b[1:] for b in bary], exps)
        vinv = _inverse(v)
        mass = _monomial_mass(exps, dim)
        massinv = _inverse(mass)
        vt = [list(c) for c in zip(*v)]
        minv = _matmul(_matmul(v, massinv), vt)
        strong, weak = [], []
        where = {a: k for k, a in enumerate(exps)}
        for r in range(dim):
            d = [[Decimal(0)] * len(exps) for _ in exps]
            for k, a in enumerate(exps):
                if a[r]:
                    lower = a[:r] + (a[r] - 1,) + a[r + 1:]
                    d[where[lower]][k] = Decimal(a[r])
            dt = [list(c) for c in zip(*d)]
            strong.append(_matmul(_matmul(v, d), vinv))
            weak.append(_matmul(_matmul(v, _matmul(massinv, _matmul(dt, mass))), vinv))
        fexps = _exponents(dim - 1, order)
        fmass = _monomial_mass(fexps, dim - 1)
        fnodes, lift = [], []
        for f in range(dim + 1):
            rest = [k for k in range(dim + 1) if k != f]
            nodes = [i for i, a in enumerate(alphas) if a[f] == 0]
            pts = [[bary[i][k] for k in rest[1:]] for i in nodes]
            fvinv = _inverse(vandermonde(pts, fexps))
            fvinvt = [list(c) for c in zip(*fvinv)]
            fm = _matmul(_matmul(fvinvt, fmass), fvinv)
            fnodes.append(nodes)
            lift.append(_matmul([[row[i] for i in nodes] for row in minv], fm))

        # face nodes in the order set by the ranks of the face's vertices: the same
        # physical point has the same place in both elements of a glued pair
        canonical = np.zeros((dim + 1, math.factorial(dim), len(fnodes[0])), dtype=np.int64)
        perms = list(itertools.permutations(range(dim)))
        for f in range(dim + 1):
            rest = [k for k in range(dim + 1) if k != f]
            for p, perm in enumerate(perms):
                by_rank = sorted(range(len(fnodes[f])), key=lambda j: tuple(
                    alphas[fnodes[f][j]][rest[k]] for k in perm))
                canonical[f, p] = by_rank

    def arr(x):
        return torch.tensor(np.array(x, dtype=np.float64), device=DEVICE)

    return dict(np_=len(exps), nfp=len(fnodes[0]), bary=arr(bary), strong=arr(strong),
                weak=arr(weak), lift=arr(lift),
                fnodes=torch.tensor(fnodes, device=DEVICE),
                canonical=torch.tensor(canonical, device=DEVICE), perms=perms)


def _box(case: dict, n: int):
    """Vertices and element vertex lists of the box mesh (cells in C order)."""
    dim = case["dim"]
    lo, hi = BOX[case["equation"]]
    axis = torch.tensor(np.linspace(lo, hi, n + 1), device=DEVICE)
    verts = torch.stack(torch.meshgrid(*[axis] * dim, indexing="ij"), -1).reshape(-1, dim)
    cell = torch.arange(n, device=DEVICE)
    base = torch.stack(torch.meshgrid(*[cell] * dim, indexing="ij"), -1).reshape(-1, 1, 1, dim)
    if dim == 3:
        split = ["000 100 010 001", "101 100 001 010", "101 011 010 001",
                 "100 010 101 110", "011 010 110 101", "011 111 101 110"]
    else:
        split = ["00 10 01", "11 01 10"]
    corner = torch.tensor([[[int(c) for c in lab] for lab in s.split()] for s in split],
                          device=DEVICE)
    pos = base + corner[None]
    idx = pos[..., 0]
    for d in range(1, dim):
        idx = idx * (n + 1) + pos[..., d]
    return verts, idx.reshape(-1, dim + 1)


def _nodes(case: dict, n: int) -> torch.Tensor:
    """(dim, Nel, Np) node coordinates."""
    verts, el = _box(case, n)
    bary = _element(case["dim"], case["order"])["bary"]
    return torch.einsum("iv,evx->xei", bary, verts[el]).contiguous()


# }}}

# {{{ inputs


def _waves(x: torch.Tensor, count: int, rng: np.random.Generator, period: float):
    """``count`` smooth fields: sums of three seeded waves, at most three per box."""
    out = []
    for _ in range(count):
        f = torch.zeros_like(x[0])
        for _ in range(3):
            k = 2.0 * math.pi / period * rng.uniform(-3.0, 3.0, size=x.shape[0])
            arg = sum(float(kd) * xd for kd, xd in zip(k, x)) + float(rng.uniform(0, 2 * math.pi))
            f += float(rng.uniform(0.3, 1.0)) * torch.cos(arg)
        out.append(f)
    return out


def _fields(case: dict, seed: int, n: int) -> torch.Tensor:
    """(nfields, Nel, Np) initial state."""
    eq, dim = case["equation"], case["dim"]
    x = _nodes(case, n)
    lo, hi = BOX[eq]
    rng = np.random.default_rng([seed, n])
    nf = NFIELDS[dim][eq]
    if eq == "wave":        # a pressure pulse on a smooth background
        f = _waves(x, nf, rng, hi - lo)
        f[0] = f[0] + torch.exp(-(x * x).sum(0) / 0.1**2)
        return torch.stack(f)
    if eq == "maxwell":
        return torch.stack(_waves(x, nf, rng, hi - lo))
    f = _waves(x, nf, rng, hi - lo)      # density, pressure and velocity of order one
    rho = 1.0 + 0.05 * f[0] + 0.1 * torch.exp(-(x * x).sum(0) / 0.2**2)
    p = 1.0 + 0.05 * f[1]
    u = [0.1 + 0.05 * v for v in f[2:]]
    energy = p / (PARAMS["euler"][0] - 1.0) + 0.5 * rho * sum(v * v for v in u)
    return torch.stack([rho, energy] + [rho * v for v in u])


def _cotangent(case: dict, seed: int) -> torch.Tensor:
    x = _nodes(case, case["n"])
    rng = np.random.default_rng([seed, 7])
    return torch.stack(_waves(x, NFIELDS[case["dim"]][case["equation"]], rng, 1.0))


def _timestep(case: dict) -> float:
    """A stable step: a fraction of a cell over the fastest signal."""
    lo, hi = BOX[case["equation"]]
    return 0.05 * (hi - lo) / (case["n"] * case["order"] ** 2)


def _receivers(case: dict, seed: int) -> np.ndarray:
    rng = np.random.default_rng([seed, 11])
    return rng.uniform(-0.9, 0.9, size=(16, 3))


def _speeds(case: dict, seed: int) -> torch.Tensor:
    """(Nel,) element wave speeds around one."""
    x = _nodes(case, case["n"]).mean(2)
    rng = np.random.default_rng([seed, 13])
    return 1.0 + 0.05 * _waves(x, 1, rng, 2.0)[0]


# }}}

# {{{ prepare and run


def prepare(case: dict, seed: int) -> dict:
    from actx_dgfem_suite_gb300.array_context import GB300DGArrayContext, stacked_state
    from actx_dgfem_suite_gb300.device_setup import DeviceBoxDiscretization
    from actx_dgfem_suite_gb300.plan import DeviceMesh, DevicePlan

    kind, eq, order, n = case["kind"], case["equation"], case["order"], case["n"]
    if kind == "rhs":
        from actx_dgfem_suite_gb300.rhs_builder import get_rhs
        actx = GB300DGArrayContext()
        rhs, args = get_rhs(eq, actx, case["dim"], order, definition="baseline", nel_1d=n,
                            device_setup=case["dim"] == 3)
        rhs.dg_operator.precision = case["precision"]
        args = args[:-1] + (stacked_state(actx, args[-1], _fields(case, seed, n)),)
        return dict(case=case, call=actx.compile(rhs), args=args)
    if kind == "ensemble":
        from actx_dgfem_suite_gb300.ensemble import Ensemble
        sizes = _member_sizes(case)
        discs = [DeviceBoxDiscretization(order, m, *BOX[eq], with_nodes=False) for m in sizes]
        ens = Ensemble(discs, eq, PARAMS[eq], case["precision"])
        q = ens.stack_states([_fields(case, seed + k, m) for k, m in enumerate(sizes)])
        ens.autotune(q, max_rel_l2=1e-5)
        ens.capture(q, torch.empty_like(q))
        return dict(case=case, ensemble=ens)
    if kind == "gradient":
        from actx_dgfem_suite_gb300.adjoint import Receivers, WaveAdjointSolver
        from actx_dgfem_suite_gb300.discretization import make_box_discretization
        disc = make_box_discretization(order, n, *BOX[eq])
        rec = Receivers(disc, _receivers(case, seed), DEVICE)
        solver = WaveAdjointSolver(disc, _timestep(case), case["steps"], rec)
        return dict(case=case, solver=solver, q0=_fields(case, seed, n),
                    c=_speeds(case, seed))
    mesh = DeviceMesh(DeviceBoxDiscretization(order, n, *BOX[eq], with_nodes=False))
    plan = DevicePlan(mesh, eq, PARAMS[eq], case["precision"])
    q = _fields(case, seed, n)
    if kind == "step":
        from actx_dgfem_suite_gb300.timestepping import LSRK45
        return dict(case=case, stepper=LSRK45(plan, _timestep(case)), q=q)
    return dict(case=case, plan=plan, q=q, x=_cotangent(case, seed))


def run(state: dict):
    kind = state["case"]["kind"]
    if kind == "rhs":
        from actx_dgfem_suite_gb300.containers import leaves
        return [d[0] for d in leaves(state["call"](*state["args"]))]
    if kind == "step":
        return state["stepper"].step(state["q"])
    if kind == "ensemble":
        return state["ensemble"].replay()
    if kind == "rhs_vjp":
        from actx_dgfem_suite_gb300.adjoint import RHSFunction
        q = state["q"].detach().requires_grad_()
        out = RHSFunction.apply(q, state["plan"])
        (grad,) = torch.autograd.grad(out, q, state["x"])
        return [out.detach(), grad]
    from actx_dgfem_suite_gb300.adjoint import WaveMisfitFunction
    q0 = state["q0"].detach().requires_grad_()
    c = state["c"].detach().requires_grad_()
    traces = WaveMisfitFunction.apply(q0, c, state["solver"])
    gq, gc = torch.autograd.grad(0.5 * (traces * traces).sum(), (q0, c))
    return [traces.detach(), gq, gc]


# }}}

# {{{ work


def work(case: dict) -> dict:
    """State in, result out and the mesh's geometry and face index read once per
    RHS; operations of the operator as written (derivative and LIFT products and
    pointwise fluxes)."""
    from actx_dgfem_suite_gb300.perf_model import flops_per_element
    dim, order, eq, kind = case["dim"], case["order"], case["equation"], case["kind"]
    npn = math.comb(order + dim, dim)
    nfp = math.comb(order + dim - 1, dim - 1)
    sizes = _member_sizes(case) if kind == "ensemble" else [case["n"]]
    nel = sum(6 * n**3 if dim == 3 else 2 * n**2 for n in sizes)
    state = 8 * NFIELDS[dim][eq] * npn
    mesh = 8 * dim * dim + 32 * (dim + 1) + 4 * (dim + 1) * nfp
    flops = flops_per_element(eq, order, dim)
    if kind == "step":        # a stage also reads and writes the residual
        per, count = 4 * state + mesh, 5
    elif kind == "rhs_vjp":   # the RHS, and q, x in and the product out
        per, count, flops = 2 * state + mesh + 3 * state + mesh, 1, 3 * flops
    elif kind == "gradient":  # two forward sweeps (recording one) and the reverse one
        per, count, flops = 3 * (4 * state + mesh) + 2 * state, 5 * case["steps"], 3 * flops
    else:
        per, count = 2 * state + mesh, 1
    return {"bytes": nel * per * count, "flops": nel * flops * count}


# }}}

# {{{ exact: the operators in plain torch, 64 bits


class _Plain:
    """Operators of one box mesh, unfused."""

    def __init__(self, case: dict, n: int):
        self.dim, self.eq = case["dim"], case["equation"]
        dim = self.dim
        el = _element(dim, case["order"])
        self.el = el
        verts, ev = _box(case, n)
        x = verts[ev]                                                # (Nel, dim+1, dim)
        nel = ev.shape[0]
        jac = (x[:, 1:] - x[:, :1]).transpose(1, 2)                  # dx/dr
        self.metric = torch.linalg.inv(jac)                          # (Nel, r, x)
        grad = torch.cat([-self.metric.sum(1, keepdim=True), self.metric], 1)
        self.scale = grad.norm(dim=2)                                # sJ/J of face f
        self.normal = -grad / self.scale[..., None]                  # (Nel, dim+1, dim)

        # face f of element e: its vertices in ascending order, and its nodes in the
        # order that the vertices' ranks set
        rest = torch.tensor([[k for k in range(dim + 1) if k != f] for f in range(dim + 1)],
                            device=DEVICE)
        fv = ev[:, rest]                                             # (Nel, F, dim)
        ranked, by = fv.sort(dim=2)
        code = torch.zeros((dim,) * dim, dtype=torch.long, device=DEVICE)
        for p, perm in enumerate(el["perms"]):
            code[perm] = p
        pid = code[tuple(by[..., k] for k in range(dim))]            # (Nel, F)
        place = el["canonical"][torch.arange(dim + 1, device=DEVICE)[None], pid]
        fnodes = el["fnodes"][None].expand(nel, -1, -1)              # (Nel, F, Nfp)
        own = torch.arange(nel, device=DEVICE)[:, None, None] * el["np_"] + fnodes
        ordered = own.gather(2, place).reshape(-1, el["nfp"])        # canonical order
        key = ranked[..., 0]
        for k in range(1, dim):
            key = key * verts.shape[0] + ranked[..., k]
        key = key.reshape(-1)
        skey, pos = key.sort()
        first = torch.nonzero(skey[1:] == skey[:-1])[:, 0]
        a, b = pos[first], pos[first + 1]
        other = ordered.clone()
        other[a], other[b] = ordered[b], ordered[a]
        boundary = torch.ones(key.shape[0], dtype=torch.bool, device=DEVICE)
        boundary[a] = False
        boundary[b] = False
        ext = torch.empty_like(own)
        ext.scatter_(2, place, other.reshape(own.shape))
        self.own, self.ext = own, ext
        self.boundary = boundary.reshape(nel, dim + 1, 1)
        self.n = [self.normal[..., d, None] for d in range(dim)]     # (Nel, F, 1)

    def traces(self, u):
        flat = u.reshape(-1)
        return flat[self.own], flat[self.ext]

    def lift(self, flux):
        f = flux * self.scale[..., None]
        return sum(f[:, k] @ self.el["lift"][k].T for k in range(self.dim + 1))

    def dref(self, u, name):
        return [u @ self.el[name][r].T for r in range(self.dim)]

    def grad(self, u, name):
        d = self.dref(u, name)
        return [sum(self.metric[:, r, x, None] * d[r] for r in range(self.dim))
                for x in range(self.dim)]

    def div(self, v, name):
        return sum(sum(self.metric[:, r, x, None] * v[x] for x in range(self.dim))
                   @ self.el[name][r].T for r in range(self.dim))

    def rhs(self, q):
        return getattr(self, self.eq)(q)

    def wave(self, q):
        dim, n, b = self.dim, self.n, self.boundary
        (c,) = PARAMS["wave"]
        ui, ue = self.traces(q[0])
        ue = torch.where(b, -ui, ue)
        vi, ve = zip(*[self.traces(q[1 + d]) for d in range(dim)])
        ve = [torch.where(b, vi[d], ve[d]) for d in range(dim)]
        fu = sum(0.5 * (vi[d] + ve[d]) * n[d] for d in range(dim)) + 0.5 * (ue - ui)
        fv = 0.5 * (ui + ue) + 0.5 * sum((ve[d] - vi[d]) * n[d] for d in range(dim))
        gu = self.grad(q[0], "weak")
        out = [self.lift(c * fu) - c * self.div(list(q[1:]), "weak")]
        out += [self.lift(c * fv * n[d]) - c * gu[d] for d in range(dim)]
        return torch.stack(out)

    def euler(self, q):
        dim, n, b = self.dim, self.n, self.boundary
        (gamma,) = PARAMS["euler"]

        def parts(s):
            rho, en, m = s[0], s[1], list(s[2:])
            u = [k / rho for k in m]
            p = (gamma - 1.0) * (en - 0.5 * sum(k * v for k, v in zip(m, u)))
            flux = [m, [(en + p) * v for v in u]]
            flux += [[m[i] * u[x] + (p if i == x else 0.0) for x in range(dim)]
                     for i in range(dim)]
            speed = torch.sqrt(sum(v * v for v in u)) + torch.sqrt(gamma * p / rho)
            return flux, speed

        qi, qe = map(list, zip(*[self.traces(q[k]) for k in range(2 + dim)]))
        mn = sum(qi[2 + d] * n[d] for d in range(dim))
        wall = [qi[0], qi[1]] + [qi[2 + d] - 2.0 * mn * n[d] for d in range(dim)]
        qe = [torch.where(b, w, e) for w, e in zip(wall, qe)]
        fi, li = parts(qi)
        fe, le = parts(qe)
        lam = torch.maximum(li, le)
        vol, _ = parts(q)
        out = []
        for k in range(2 + dim):
            fn = sum(0.5 * (fi[k][x] + fe[k][x]) * n[x] for x in range(dim))
            fn = fn - 0.5 * lam * (qe[k] - qi[k])
            out.append(self.div(vol[k], "weak") - self.lift(fn))
        return torch.stack(out)

    def maxwell(self, q):
        b = self.boundary
        alpha, eps, mu = PARAMS["maxwell"]
        z = math.sqrt(mu / eps)
        y = 1.0 / z
        zero = torch.zeros_like(q[0])
        full = list(q) if self.dim == 3 else [zero, zero, q[0], q[1], q[2], zero]
        n = self.n + [torch.zeros_like(self.n[0])] * (3 - self.dim)

        def cross(a, c):
            return [a[1] * c[2] - a[2] * c[1], a[2] * c[0] - a[0] * c[2],
                    a[0] * c[1] - a[1] * c[0]]

        def curl(w):
            d = [self.grad(f, "strong") + [zero] * (3 - self.dim) for f in w]
            return [d[2][1] - d[1][2], d[0][2] - d[2][0], d[1][0] - d[0][1]]

        je, jh = [], []
        for f in full[:3]:
            i, e = self.traces(f)
            je.append(torch.where(b, -2.0 * i, e - i))
        for f in full[3:]:
            i, e = self.traces(f)
            jh.append(torch.where(b, torch.zeros_like(i), e - i))
        ne, nh = cross(n, je), cross(n, jh)
        fe = cross(n, [z * jh[k] - alpha * ne[k] for k in range(3)])
        fh = cross(n, [y * je[k] + alpha * nh[k] for k in range(3)])
        ch, ce = curl(full[3:]), curl(full[:3])
        want = range(6) if self.dim == 3 else (2, 3, 4)
        out = []
        for k in want:
            if k < 3:
                out.append((ch[k] + self.lift(fe[k] / (z + z))) / eps)
            else:
                out.append((-ce[k - 3] - self.lift(fh[k - 3] / (y + y))) / mu)
        return torch.stack(out)


_RKA = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
        -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
_RKB = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
        1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
        2277821191437.0 / 14882151754819.0)


def _lsrk_step(rhs, q, dt):
    """Carpenter & Kennedy's five-stage low-storage step."""
    res = torch.zeros_like(q)
    for a, b in zip(_RKA, _RKB):
        res = a * res + dt * rhs(q)
        q = q + b * res
    return q


def exact(case: dict, seed: int):
    kind, n = case["kind"], case["n"]
    if kind == "ensemble":
        with torch.no_grad():
            return torch.cat([_Plain(case, m).rhs(_fields(case, seed + k, m))
                              for k, m in enumerate(_member_sizes(case))], dim=1)
    plain = _Plain(case, n)
    q = _fields(case, seed, n)
    if kind == "rhs":
        with torch.no_grad():
            return list(plain.rhs(q))
    if kind == "step":
        with torch.no_grad():
            return _lsrk_step(plain.rhs, q, _timestep(case))
    q.requires_grad_()
    if kind == "rhs_vjp":
        out = plain.rhs(q)
        (grad,) = torch.autograd.grad(out, q, _cotangent(case, seed))
        return [out.detach(), grad]
    c = _speeds(case, seed).requires_grad_()
    pts = torch.tensor(_receivers(case, seed), device=DEVICE)
    weights, elems = _point_weights(case, pts)
    w, traces = q, []
    for _ in range(case["steps"]):
        w = _lsrk_step(lambda s: c[:, None] * plain.rhs(s), w, _timestep(case))
        traces.append((w[0, elems] * weights).sum(1))
    traces = torch.stack(traces)
    gq, gc = torch.autograd.grad(0.5 * (traces * traces).sum(), (q, c))
    return [traces.detach(), gq, gc]


def _point_weights(case: dict, pts: torch.Tensor):
    """Interpolation weights of points in the elements that hold them."""
    el = _element(3, case["order"])
    verts, ev = _box(case, case["n"])
    x = verts[ev]
    inv = torch.linalg.inv((x[:, 1:] - x[:, :1]).transpose(1, 2))
    exps = torch.tensor(_exponents(3, case["order"]), device=DEVICE)

    def powers(r):
        return (r[:, None, :] ** exps[None]).prod(2)

    vinv = torch.linalg.inv(powers(el["bary"][:, 1:]))
    elems, ref = [], []
    for p in pts:
        r = torch.einsum("erx,ex->er", inv, p - x[:, 0])
        inside = ((r >= -1e-10).all(1)) & (r.sum(1) <= 1 + 1e-10)
        e = int(torch.nonzero(inside)[0, 0])
        elems.append(e)
        ref.append(r[e])
    return powers(torch.stack(ref)) @ vinv, torch.tensor(elems, device=DEVICE)


# }}}
