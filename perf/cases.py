"""What this package is timed on: marches, batched sweeps, residuals and adjoint work, by their public calls.

A case is a dict of plain values.  ``path`` says which call it is:

* ``march``     ``B200Backend.run``: a chunk of steps of one solve, host state in and out, as
                ``march.solve`` (and the host solver this backend plugs into) calls it;
* ``batch``     ``BatchSolver``: a design sweep's members marched together for ``steps`` steps (the
                observables, taken once after tens of thousands of steps, are left out);
* ``stage``     ``BatchSolver`` with one member: a device-resident step of one large mesh of random
                admissible states, about half of whose elements the limiter works on;
* ``residual``  ``AdjointModel.residual``: one residual of a device-resident state;
* ``gradient``  ``ResidualFunction`` and ``torch.autograd.grad``: the residual and its products with
                respect to the state, the node coordinates and the back pressure;
* ``adjoint``   ``AdjointMarch.solve``: RK4 steps of the discrete adjoint.

Nozzle cases draw the design point (area ratio, back pressure) from the seed, so every seed is another
nozzle of the same size.  :func:`exact` evaluates the same mathematics in plain 64-bit torch.
"""

from __future__ import annotations

import functools
import importlib
import math
from types import SimpleNamespace

import numpy as np
import torch

PACKAGE = "2d_nozzle_b200"


def _pkg(name):
    return importlib.import_module(f"{PACKAGE}.{name}")


# ------------------------------------------------------------------ the cases
def listed():
    nozzle = {"nx": 14, "nr": 5, "q": 1, "limiter": "positivity"}  # the case builder's base mesh
    return [
        # The quick start's coarsest mesh: linear triangles, Roe; 150 tiny stages, so launches and
        # latency are all there is.
        {"name": "march tri p1 140", "path": "march", "element": "tri", "order": 1, "refine": 0, "flux": "roe",
         "steps": 50, **nozzle},
        # The forward solve of a shape gradient: quadratic triangles, AUSM+-up.
        {"name": "march tri p2 2240", "path": "march", "element": "tri", "order": 2, "refine": 2, "flux": "ausmup",
         "steps": 50, **nozzle},
        # The largest single nozzle solve of the sweeps: cubic quadrilaterals, HLLC.
        {"name": "march quad p3 4480", "path": "march", "element": "quad", "order": 3, "refine": 3, "flux": "hllc",
         "steps": 50, **nozzle},
        # The other limiter: Superbee slopes, then positivity.
        {"name": "march tri p2 superbee 2240", "path": "march", "element": "tri", "order": 2, "refine": 2,
         "flux": "hllc", "steps": 50, **{**nozzle, "limiter": "superbee"}},
        # Orders above 3 (the generic kernels).
        {"name": "march tri p4 2240", "path": "march", "element": "tri", "order": 4, "refine": 2, "flux": "roe",
         "steps": 20, **nozzle},
        # Curved (quadratic-geometry) elements, also on the generic kernels.
        {"name": "march quad p2 curved 4480", "path": "march", "element": "quad", "order": 2, "refine": 3,
         "flux": "roe", "steps": 20, **{**nozzle, "q": 2}},
        # The design sweep: orders 1..3, refinements 1..3, triangles and quadrilaterals in equal parts,
        # 72 members (211 680 elements) in six buckets -- the headline workload at its usual size.
        {"name": "batch sweep 72", "path": "batch", "members": 72, "flux": "hllc", "steps": 51,
         **{**nozzle, "element": "mixed", "order": 0, "refine": 0}},
        # One limited SSP-RK3 step of a large mesh of cubic triangles (the stage microbenchmark).
        {"name": "stage tri p3 500k", "path": "stage", "element": "tri", "order": 3, "nx": 500, "nr": 500,
         "flux": "hllc", "steps": 1},
        # One residual of the million-element microbenchmark: the largest call.
        {"name": "residual tri p3 1M", "path": "residual", "element": "tri", "order": 3, "nx": 1000, "nr": 500,
         "flux": "roe"},
        # The differentiable residual on quadrilaterals: forward, state, coordinate and pressure products.
        {"name": "gradient quad p2 17920", "path": "gradient", "element": "quad", "order": 2, "refine": 4,
         "flux": "roe", **nozzle},
        # One design's adjoint march (one check interval of RK4 steps).
        {"name": "adjoint tri p2 2240", "path": "adjoint", "element": "tri", "order": 2, "refine": 2,
         "flux": "ausmup", "steps": 100, **nozzle},
        # The adjoint march at the size of a 64-member gradient batch.
        {"name": "adjoint tri p2 143k", "path": "adjoint", "element": "tri", "order": 2, "refine": 5,
         "flux": "ausmup", "steps": 10, **nozzle},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh_size(rng, element, lo, hi):
    """nx, nr of a channel about three times as long as high with lo..hi elements (odd sizes included)."""
    cells = _log_int(rng, lo, hi) / (2 if element == "tri" else 1)
    nr = max(2, int(round(math.sqrt(cells / 3.0) * rng.uniform(0.8, 1.25))))
    return max(4, int(cells / nr)), nr


def draw(rng):
    path = rng.choice(["march", "march", "march", "curved", "batch", "stage", "residual", "gradient", "adjoint"])
    element = rng.choice(["tri", "quad"])
    flux = rng.choice(["roe", "hllc", "ausmup"])
    order = rng.choice([1, 2, 3])
    case = {"path": path, "element": element, "order": order, "flux": flux}
    if path == "march":
        case["order"] = order = rng.choice([0, 1, 1, 2, 2, 3, 3])
        limiter = rng.choice(["positivity", "positivity", "superbee", "none"])
        case["nx"], case["nr"] = _mesh_size(rng, element, 120, 12000)
        case.update(refine=0, q=1, limiter=limiter, steps=rng.randint(10, 60))
    elif path == "curved":  # the generic kernels: curved elements, or orders above 3
        q = rng.choice([1, 2])
        case.update(path="march", q=q, order=rng.choice([4, 5] if q == 1 and element == "tri" else [4] if q == 1 else [1, 2, 3]))
        case["nx"], case["nr"] = _mesh_size(rng, element, 120, 4000)
        case.update(refine=0, limiter=rng.choice(["positivity", "superbee"]), steps=rng.randint(5, 25))
    elif path == "batch":
        nx, nr = rng.randint(9, 17), rng.randint(3, 6)
        case.update(members=_log_int(rng, 3, 48), steps=rng.randint(11, 51), nx=nx, nr=nr, q=1, limiter="positivity",
                    element="mixed", order=0, refine=0)
    elif path == "stage":
        case["nx"], case["nr"] = _mesh_size(rng, element, 20000, 400000 if element == "tri" else 200000)
        case["steps"] = 1
    elif path == "residual":
        case["nx"], case["nr"] = _mesh_size(rng, element, 1000, 900000 if element == "tri" else 400000)
    else:
        case["nx"], case["nr"] = _mesh_size(rng, element, 400, 30000)
        case.update(refine=0, q=1, limiter="positivity")
        if path == "adjoint":
            elements = case["nx"] * case["nr"] * (2 if element == "tri" else 1)
            case["steps"] = max(5, min(100, 200000 // elements))
    return case


# ------------------------------------------------------------------ what a program has in hand
def _options(case, **kw):
    """The plain solve's options: its cfl of 0.5 keeps every element type and order stable from the initial
    state, where the default cfl lets quadrilaterals of order 2 and 3 blow any rounding up within tens of steps."""
    return _pkg("config").SolverOptions(cfl=0.5, limiter=case.get("limiter", "positivity"), tolerance=1e-10,
                                        print_interval=0, **kw)


def _design(rng):
    """A shock-free design point: the over-expanded nozzles of the sweep's range."""
    return rng.uniform(1.5, 4.0), rng.uniform(0.1, 0.2)


def _nozzle(case, seed, lean=False, contour="smooth"):
    ar, pb = _design(np.random.default_rng([int(seed), 17]))
    flow = _pkg("config").FlowConditions(flux=case["flux"], back_pressure_ratio=pb)
    return _pkg("nozzle").build_case(element=case["element"], order=case["order"], refine=case["refine"], nx=case["nx"],
                                     nr=case["nr"], geometry_order=case["q"], area_ratio=ar, contour=contour, flow=flow,
                                     options=_options(case), lean=lean)


@functools.lru_cache(maxsize=2)
def _rectangle(element, order, nx, nr):
    """Operators of the unit rectangle: a microbenchmark keeps its mesh and changes the states."""
    topo, xf, rf = _pkg("mesh").channel_topology(element, nx=nx, nr=nr)
    return _pkg("operators").build_operators(topo, _pkg("mesh").rectangle_coords(xf, rf), order, lean=True)


def _random_state(n_elem, n_basis, seed, device="cuda"):
    """(E, NP, 4): density lognormal(0, 0.3), Mach U[0.2, 3] in a random direction, pressure lognormal(0, 0.5)."""
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed))
    kw = {"generator": gen, "dtype": torch.float64, "device": device}
    shape, g = (n_elem, n_basis), 1.4
    rho = torch.exp(0.3 * torch.randn(shape, **kw))
    mach = 0.2 + 2.8 * torch.rand(shape, **kw)
    ang = 2.0 * math.pi * torch.rand(shape, **kw)
    p = torch.exp(0.5 * torch.randn(shape, **kw))
    a = torch.sqrt(g * p / rho)
    vx, vy = mach * a * torch.cos(ang), mach * a * torch.sin(ang)
    return torch.stack([rho, rho * vx, rho * vy, p / (g - 1.0) + 0.5 * rho * (vx * vx + vy * vy)], -1)


def _members(case, seed):
    """A sweep's members: every (element, order, refinement) class in turn, each at its own design point."""
    rng = np.random.default_rng([int(seed), 5])
    classes = [(e, p, r) for r in (1, 2, 3) for p in (1, 2, 3) for e in ("tri", "quad")]
    opts = _options(case, max_iterations=case["steps"])
    out = []
    for k in range(case["members"]):
        element, order, refine = classes[(k * 7) % len(classes)] if case["members"] < len(classes) else classes[k % len(classes)]
        ar, pb = _design(rng)
        flow = _pkg("config").FlowConditions(flux=case["flux"], back_pressure_ratio=pb)
        cs = _pkg("nozzle").build_case(element=element, order=order, refine=refine, nx=case["nx"], nr=case["nr"],
                                       area_ratio=ar, contour="bell", flow=flow, options=opts, lean=True)
        out.append(_pkg("batch").Instance(cs.operators, flow, opts, None, cs.geometry.length, cs.geometry))
    return out


def _flow_state(case, cs):
    """The (E, NP, 4) device state of a nozzle some steps into its march: what an adjoint is linearised about."""
    bk = _pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
    U, _ = bk.run(bk.initial_state(cs.geometry), 20, bk.scheme)
    return torch.as_tensor(U, device="cuda")


def _residual_parts(case, seed):
    ops = _rectangle(case["element"], case["order"], case["nx"], case["nr"])
    flow = _pkg("config").FlowConditions(flux=case["flux"])
    return ops, flow, _options(case), _random_state(int(ops.n_elem), int(ops.ref.n_basis), seed)


def prepare(case, seed):
    path = case["path"]
    s = SimpleNamespace(path=path, case=case)
    if path == "march":
        cs = _nozzle(case, seed)
        s.backend = _pkg("backend").B200Backend(cs.operators, cs.flow, cs.options)
        s.U0 = cs.initial_state()
    elif path == "batch":
        s.solver = _pkg("batch").BatchSolver(_members(case, seed))
    elif path == "stage":
        ops, flow, _, U = _residual_parts(case, seed)
        # a random state's residual says nothing about convergence: the march's tests are out of the way
        opts = _options(case, max_iterations=case["steps"], divergence_factor=1e300, stall_ratio=2.0)
        s.solver = _pkg("batch").BatchSolver([_pkg("batch").Instance(ops, flow, opts, U.cpu().numpy())])
    elif path == "residual":
        ops, flow, opts, U = _residual_parts(case, seed)
        s.model = _model(ops, flow, opts)
        s.U = _pkg("adjoint").to_soa(U)
    else:
        ad = _pkg("adjoint")
        cs = _nozzle(case, seed)
        U = _flow_state(case, cs)
        s.model = _model(cs.operators, cs.flow, cs.options)
        s.U = ad.to_soa(U)
        if path == "gradient":
            s.X = torch.as_tensor(cs.node_coords, device="cuda")
            s.p_back = torch.tensor(float(cs.flow.back_pressure), dtype=torch.float64, device="cuda")
            s.lam = _cotangent(s.U, seed)
        else:
            s.march = ad.AdjointMarch(s.model, s.U, ad.to_soa(_thrust_seed(s.model, U)), cs.options.cfl)
    return s


def _model(ops, flow, opts):
    """The device model of a mesh; quadrilaterals of a lean build get their inverse mass matrices here."""
    if ops.inv_mass is None and ops.ref.kind != "tri":
        ops = _pkg("operators").build_operators(ops.topology, ops.node_coords, ops.ref.order)
    return _pkg("adjoint").AdjointModel(ops, flow, opts)


def _cotangent(like, seed):
    gen = torch.Generator(device=like.device)
    gen.manual_seed(int(seed) + 1)
    return torch.randn(like.shape, generator=gen, dtype=torch.float64, device=like.device)


def _thrust_seed(model, U):
    """d(thrust)/dU of the (E, NP, 4) state."""
    Ug = U.clone().requires_grad_(True)
    J = _pkg("adjoint").objective_value(model, Ug, model.X0, "thrust", {})
    return torch.autograd.grad(J, Ug)[0]


# ------------------------------------------------------------------ one pass
def run(s):
    if s.path == "march":
        U, res = s.backend.run(s.U0, s.case["steps"], s.backend.scheme)
        return {"U": U, "residual": res}
    if s.path == "batch":
        s.solver.reset()
        s.solver.run()
        res = s.solver.results(with_state=False)
        return {"states": [S[0] for _, S in s.solver.buffers],  # every member's state, bucket by bucket
                "residuals": np.array([r.residual for r in res]), "iterations": np.array([r.iterations for r in res])}
    if s.path == "stage":
        s.solver.reset()
        s.solver.run()
        return {"U": s.solver.buffers[0][1][0], "residual": s.solver.t["res"]}
    if s.path == "residual":
        R, wave = s.model.residual(s.U)
        return {"R": R, "wave": wave}
    if s.path == "gradient":
        U, X, pb = (t.detach().clone().requires_grad_(True) for t in (s.U, s.X, s.p_back))
        R = _pkg("adjoint").ResidualFunction(s.model, U, X, pb)
        gU, gX, gpb = torch.autograd.grad(R, (U, X, pb), s.lam)
        return {"R": R.detach(), "gU": gU, "gX": gX, "gpb": gpb}
    n = s.case["steps"]
    lam, rel, its, _ = s.march.solve(tolerance=1e-8, max_iterations=n, check_interval=n)
    return {"lam": lam, "rel": rel, "iterations": its}


# ------------------------------------------------------------------ what a pass cannot do without
def _sizes(element, order, q=1):
    """Basis functions, volume points, face points, faces and edge nodes of one element."""
    n = (2 * order * q + 1 + 2) // 2
    if element == "tri":
        return (order + 1) * (order + 2) // 2, n * n if order > 0 else 1, n, 3, order + 1
    return (order + 1) ** 2, n * n, n, 4, order + 1


def _element_work(element, order, q, stage):
    """(bytes, flops) of one element's residual (or stage): its state read and result written once, geometry,
    connectivity, one edge record per edge; the contractions, one Euler flux per volume point and half a
    Riemann flux per face point (each edge's flux is needed once)."""
    NP, NQV, NQF, NF, NE = _sizes(element, order, q)
    S = NP * 32
    b = 2 * S + (40 if element == "tri" else 64) + 12 * NF + 16 * NF + 8
    f = NQV * (8 * NP + 60 + 16 * NP) + NF * NQF * (8 * NE + 80 + 8 * NE)
    if stage:  # two of three stages read the step's start too; the local step; the inverse mass
        b += 2 * S / 3 + 16 + (0 if element == "tri" and q == 1 else 8 * NP * NP)
        f += 8 * NP * NP + 24 * NP
    return b, f


def work(case):
    path = case["path"]
    if path == "batch":
        classes = [(e, p, r) for r in (1, 2, 3) for p in (1, 2, 3) for e in ("tri", "quad")]
        B = F = 0.0
        for k in range(case["members"]):
            e, p, r = classes[(k * 7) % 18] if case["members"] < 18 else classes[k % 18]
            b, f = _element_work(e, p, 1, True)
            n = case["nx"] * case["nr"] * 4 ** r * (2 if e == "tri" else 1) * 3 * case["steps"]
            B, F = B + b * n, F + f * n
        return {"bytes": B, "flops": F}
    e, p = case["element"], case["order"]
    E = case["nx"] * case["nr"] * 4 ** case.get("refine", 0) * (2 if e == "tri" else 1)
    if path in ("march", "stage"):
        b, f = _element_work(e, p, case.get("q", 1), True)
        n = case["steps"] * (3 if p > 0 else 1)
        io = 2 * E * _sizes(e, p, 1)[0] * 32 if path == "march" else 0
        return {"bytes": b * E * n + io, "flops": f * E * n}
    b, f = _element_work(e, p, 1, False)
    NP = _sizes(e, p)[0]
    if path == "residual":
        return {"bytes": b * E, "flops": f * E}
    vb, vf = b + NP * 32, 3 * f  # a product reads the adjoint state too; transposed contractions and Jacobians
    if path == "gradient":
        return {"bytes": (b + 2 * vb) * E, "flops": (f + 2 * vf) * E}
    n = 4 * case["steps"]
    return {"bytes": (vb + 2 * NP * 32) * E * n, "flops": (vf + 8 * NP * NP) * E * n}


# ------------------------------------------------------------------ the same in plain 64-bit torch
class _Plain:
    """The nodal DG residual, its limiters and its march in torch, from a mesh and its reference tables."""

    FLOOR = 1e-10

    def __init__(self, ops, flow, opts, device="cuda"):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(np.asarray(a)), device=device)  # noqa: E731
        ref, topo = ops.ref, ops.topology
        ed = topo.edges
        self.flow, self.opts, self.order, self.g = flow, opts, ref.order, flow.gamma
        self.phi, self.w, self.wf = t(ref.phi_vol), t(ref.w_vol), t(ref.w_face)
        self.dxi, self.deta = t(ref.dphi_dxi_vol) * self.w, t(ref.dphi_deta_vol) * self.w
        self.gxi, self.geta, self.gsig = t(ref.dgeom_dxi_vol), t(ref.dgeom_deta_vol), t(ref.dgeom_dsigma_face)
        self.nodes = t(topo.elem_nodes).long()
        self.pf = t(ref.phi_face)  # (side, face, node, point)
        self.face_edge, self.side = t(ed.face_edge).long(), t(ed.face_side).long()
        self.ie, self.if_ = t(ed.iedge_elem).long(), t(ed.iedge_face).long()
        self.be, self.bf = t(ed.bedge_elem).long(), t(ed.bedge_face).long()
        self.tags, self.ni = ed.tag_slices, int(ed.n_interior)
        self.X = t(np.asarray(ops.node_coords, float))
        self.p_back = torch.tensor(float(flow.back_pressure), dtype=torch.float64, device=device)
        self.geometry(self.X)

    def geometry(self, X):
        Xe = X[self.nodes]
        self.xxi, self.xeta = Xe[..., 0] @ self.gxi, Xe[..., 0] @ self.geta
        self.yxi, self.yeta = Xe[..., 1] @ self.gxi, Xe[..., 1] @ self.geta
        wdet = self.w * (self.xxi * self.yeta - self.xeta * self.yxi)
        self.area = wdet.sum(1)
        self.mean_w = (wdet @ self.phi.T) / self.area[:, None]
        self.wdet = wdet
        own = torch.cat([self.ie[:, 0], self.be]), torch.cat([self.if_[:, 0], self.bf])
        tan = torch.zeros(len(own[0]), self.gsig.shape[2], 2, dtype=X.dtype, device=X.device)
        for f in range(self.gsig.shape[0]):
            k = torch.nonzero(own[1] == f).squeeze(1)
            tan = tan.index_copy(0, k, torch.einsum("nq,end->eqd", self.gsig[f], Xe[own[0][k]]))
        self.jac = torch.sqrt(tan[..., 0] ** 2 + tan[..., 1] ** 2)
        self.nx, self.ny = tan[..., 1] / self.jac, -tan[..., 0] / self.jac
        self.length = self.jac @ self.wf

    @functools.cached_property
    def chol(self):
        outer = (self.phi[:, None] * self.phi[None]).reshape(-1, self.phi.shape[1])
        n = self.phi.shape[0]
        return torch.linalg.cholesky((self.wdet @ outer.T).reshape(-1, n, n))

    def primitives(self, U):
        rho = torch.clamp(U[..., 0], min=self.FLOOR)
        vx, vy = U[..., 1] / rho, U[..., 2] / rho
        p = torch.clamp((self.g - 1.0) * (U[..., 3] - 0.5 * rho * (vx * vx + vy * vy)), min=self.FLOOR)
        return rho, vx, vy, p, (U[..., 3] + p) / rho

    def normal_flux(self, U, nx, ny):
        rho, vx, vy, p, H = self.primitives(U)
        vn = vx * nx + vy * ny
        return torch.stack([rho * vn, rho * vx * vn + p * nx, rho * vy * vn + p * ny, rho * H * vn], -1)

    def roe_average(self, L, R):
        sL, sR = torch.sqrt(L[0]), torch.sqrt(R[0])
        return [(sL * L[k] + sR * R[k]) / (sL + sR) for k in (1, 2, 4)]

    def roe(self, UL, UR, nx, ny):
        g, L, R = self.g, self.primitives(UL), self.primitives(UR)
        vx, vy, H = self.roe_average(L, R)
        q2, vn = vx * vx + vy * vy, vx * nx + vy * ny
        c = torch.sqrt(torch.clamp((g - 1.0) * (H - 0.5 * q2), min=self.FLOOR))
        lam = [(vn + c).abs(), (vn - c).abs(), vn.abs()]
        smax, eps = torch.maximum(lam[0], lam[1]), self.flow.entropy_fix * c
        l1, l2, l3 = (torch.where(x < eps, (x * x + eps * eps) / (2.0 * eps), x) for x in lam)
        d = [UR[..., k] - UL[..., k] for k in range(4)]
        G1 = (g - 1.0) * (0.5 * q2 * d[0] - vx * d[1] - vy * d[2] + d[3])
        G2 = -vn * d[0] + d[1] * nx + d[2] * ny
        s1, s2 = 0.5 * (l1 + l2), 0.5 * (l1 - l2)
        C1 = G1 / (c * c) * (s1 - l3) + G2 / c * s2
        C2 = G1 / c * s2 + (s1 - l3) * G2
        D = torch.stack([l3 * d[0] + C1, l3 * d[1] + C1 * vx + C2 * nx, l3 * d[2] + C1 * vy + C2 * ny,
                         l3 * d[3] + C1 * H + C2 * vn], -1)
        return 0.5 * (self.normal_flux(UL, nx, ny) + self.normal_flux(UR, nx, ny)) - 0.5 * D, smax

    def hllc(self, UL, UR, nx, ny):
        g, L, R = self.g, self.primitives(UL), self.primitives(UR)
        vx, vy, H = self.roe_average(L, R)
        at = torch.sqrt(torch.clamp((g - 1.0) * (H - 0.5 * (vx * vx + vy * vy)), min=self.FLOOR))
        vt = vx * nx + vy * ny
        vnL, vnR = L[1] * nx + L[2] * ny, R[1] * nx + R[2] * ny
        aL, aR = (torch.sqrt(torch.clamp(g * K[3] / K[0], min=self.FLOOR)) for K in (L, R))
        SL, SR = torch.minimum(vnL - aL, vt - at), torch.maximum(vnR + aR, vt + at)
        mL, mR = L[0] * (SL - vnL), R[0] * (SR - vnR)
        dm = torch.where((mR - mL).abs() > self.FLOOR, mR - mL, self.FLOOR)
        SM = (vnR * mR - vnL * mL + L[3] - R[3]) / dm

        def guard(x):
            return torch.where(x.abs() > self.FLOOR, x, self.FLOOR)

        def star(U, K, vn, S):
            rs = K[0] * (S - vn) / guard(S - SM)
            E = U[..., 3] / K[0] + (SM - vn) * (SM + K[3] / guard(K[0] * (S - vn)))
            Us = torch.stack([rs, rs * (K[1] + (SM - vn) * nx), rs * (K[2] + (SM - vn) * ny), rs * E], -1)
            return S[..., None] * (Us - U)

        FL, FR = self.normal_flux(UL, nx, ny), self.normal_flux(UR, nx, ny)
        inner = torch.where((SM >= 0.0)[..., None], FL + star(UL, L, vnL, SL), FR + star(UR, R, vnR, SR))
        F = torch.where((SL >= 0.0)[..., None], FL, torch.where((SR <= 0.0)[..., None], FR, inner))
        return F, torch.maximum(SL.abs(), SR.abs())

    def ausmup(self, UL, UR, nx, ny):
        beta, alpha, kp, ku = 0.125, 0.1875, 0.4, 0.2
        g, L, R = self.g, self.primitives(UL), self.primitives(UR)
        vnL, vnR = L[1] * nx + L[2] * ny, R[1] * nx + R[2] * ny
        aL, aR = torch.sqrt(g * L[3] / L[0]), torch.sqrt(g * R[3] / R[0])
        a, rho = 0.5 * (aL + aR), 0.5 * (L[0] + R[0])
        mL, mR = vnL / a, vnR / a

        def split(m, s):  # the Mach and pressure polynomials of sign s
            m2, o2 = 0.25 * s * (m + s) ** 2, -0.25 * s * (m - s) ** 2
            m4 = torch.where(m.abs() >= 1.0, 0.5 * (m + s * m.abs()), m2 * (1.0 - s * 16.0 * beta * o2))
            p5 = torch.where(m.abs() >= 1.0, 0.5 * (1.0 + s * torch.sign(m)), m2 * ((s * 2.0 - m) - s * 16.0 * alpha * m * o2))
            return m4, p5

        (m4L, p5L), (m4R, p5R) = split(mL, 1.0), split(mR, -1.0)
        mb2 = 0.5 * (mL * mL + mR * mR)
        uh = a * (m4L + m4R) + kp * torch.clamp(1.0 - mb2, min=0.0) * (L[3] - R[3]) / (rho * a)
        ph = p5L * L[3] + p5R * R[3] + ku * p5L * p5R * rho * a * (vnL - vnR)
        PL, PR = (torch.stack([K[0], K[0] * K[1], K[0] * K[2], U[..., 3] + K[3]], -1) for K, U in ((L, UL), (R, UR)))
        F = 0.5 * uh[..., None] * (PL + PR) - 0.5 * uh.abs()[..., None] * (PR - PL)
        z = torch.zeros_like(ph)
        return F + torch.stack([z, ph * nx, ph * ny, z], -1), torch.maximum(vnL.abs() + aL, vnR.abs() + aR)

    def wall(self, U, nx, ny):
        rho = torch.clamp(U[..., 0], min=self.FLOOR)
        vx, vy = U[..., 1] / rho, U[..., 2] / rho
        vn = vx * nx + vy * ny
        vt2 = (vx - vn * nx) ** 2 + (vy - vn * ny) ** 2
        p = torch.clamp((self.g - 1.0) * (U[..., 3] - 0.5 * rho * vt2), min=self.FLOOR)
        z = torch.zeros_like(p)
        return torch.stack([z, p * nx, p * ny, z], -1), torch.sqrt(self.g * p / rho)

    def inflow(self, U, nx, ny):
        g, fl = self.g, self.flow
        at2 = g * fl.Rgas * fl.total_temperature
        rho, vx, vy, p, _ = self.primitives(U)
        beta = ((vx * nx + vy * ny + 2.0 * torch.sqrt(g * p / rho) / (g - 1.0)) / math.sqrt(at2)) ** 2
        cs, sn = math.cos(fl.inflow_angle), math.sin(fl.inflow_angle)
        nd = nx * cs + ny * sn
        qa, qb = 0.5 * (g - 1.0) * beta - nd * nd, -4.0 * nd / (g - 1.0)
        qa = torch.where(qa.abs() < 1e-12, torch.where(qa >= 0, 1e-12, -1e-12), qa)
        sq = torch.sqrt(torch.clamp(qb * qb - 4.0 * qa * (beta - (2.0 / (g - 1.0)) ** 2), min=0.0))
        r1, r2 = (-qb + sq) / (2.0 * qa), (-qb - sq) / (2.0 * qa)
        M = torch.minimum(torch.where(r1 >= 0.0, r1, 1e30), torch.where(r2 >= 0.0, r2, 1e30))
        M = torch.clamp(torch.where(M > 0.5e30, 0.0, M), 0.0, 1.0)
        fac = 1.0 + 0.5 * (g - 1.0) * M * M
        a = torch.sqrt(at2 / fac)
        rho = g * fl.total_pressure / at2 * fac ** (-1.0 / (g - 1.0))
        ux, uy = M * a * cs, M * a * sn
        vn, p = ux * nx + uy * ny, rho * a * a / g
        F = torch.stack([rho * vn, rho * ux * vn + p * nx, rho * uy * vn + p * ny, rho * at2 / (g - 1.0) * vn], -1)
        return F, vn.abs() + a

    def outflow(self, U, nx, ny):
        g, pb = self.g, self.p_back
        rho, vx, vy, p, _ = self.primitives(U)
        a, vn = torch.sqrt(g * p / rho), vx * nx + vy * ny
        rb = rho * (pb / p) ** (1.0 / g)
        ab = torch.sqrt(g * pb / rb)
        vb = vn + 2.0 / (g - 1.0) * (a - ab)
        ux, uy = vx - vn * nx + vb * nx, vy - vn * ny + vb * ny
        Us = torch.stack([rb, rb * ux, rb * uy, rb * (pb / ((g - 1.0) * rb) + 0.5 * (ux * ux + uy * uy))], -1)
        Ub = torch.where((vn / a >= 1.0)[..., None], U, Us)
        ro, uo, vo, po, _ = self.primitives(Ub)
        return self.normal_flux(Ub, nx, ny), (uo * nx + vo * ny).abs() + torch.sqrt(g * po / ro)

    def trace(self, U, side, elem, face):
        out = torch.zeros(len(elem), self.pf.shape[3], 4, dtype=U.dtype, device=U.device)
        for f in range(self.pf.shape[1]):
            k = torch.nonzero(face == f).squeeze(1)
            out = out.index_copy(0, k, torch.einsum("iq,kis->kqs", self.pf[side, f], U[elem[k]]))
        return out

    def residual(self, U):
        ni = self.ni
        UL, UR = self.trace(U, 0, self.ie[:, 0], self.if_[:, 0]), self.trace(U, 1, self.ie[:, 1], self.if_[:, 1])
        parts = [getattr(self, self.flow.flux)(UL, UR, self.nx[:ni], self.ny[:ni])]
        Ub = self.trace(U, 0, self.be, self.bf)
        kinds = {_pkg("mesh").INFLOW: self.inflow, _pkg("mesh").OUTFLOW: self.outflow}
        for tag, sl in sorted(self.tags.items(), key=lambda kv: kv[1].start):
            k = slice(ni + sl.start, ni + sl.stop)
            parts.append(kinds.get(tag, self.wall)(Ub[sl], self.nx[k], self.ny[k]))
        F, speed = torch.cat([x[0] for x in parts]), torch.cat([x[1] for x in parts])
        rho, vx, vy, p, H = self.primitives(torch.einsum("iq,eis->eqs", self.phi, U))
        Fx = torch.stack([rho * vx, rho * vx * vx + p, rho * vx * vy, rho * vx * H], -1)
        Fy = torch.stack([rho * vy, rho * vx * vy, rho * vy * vy + p, rho * vy * H], -1)
        a = self.yeta[..., None] * Fx - self.xeta[..., None] * Fy
        b = self.xxi[..., None] * Fy - self.yxi[..., None] * Fx
        R = -(torch.einsum("iq,eqs->eis", self.dxi, a) + torch.einsum("iq,eqs->eis", self.deta, b))
        fw = F * (self.jac * self.wf)[..., None]
        for f in range(self.pf.shape[1]):
            part = torch.zeros_like(R)
            for sd in (0, 1):
                k = torch.nonzero(self.side[:, f] == sd).squeeze(1)
                lift = torch.einsum("iq,eqs->eis", self.pf[sd, f], fw[self.face_edge[k, f]])
                part = part.index_copy(0, k, lift if sd == 0 else -lift)
            R = R + part
        wave = (speed.max(1).values * self.length)[self.face_edge].sum(1)
        return R, wave

    def rate(self, U):
        R, wave = self.residual(U)
        return -torch.cholesky_solve(R, self.chol), wave

    def face_values(self, U):
        """(E, face, point, 4): every element's own trace on its own faces."""
        basis = self.pf[self.side, torch.arange(self.pf.shape[1], device=U.device)[None, :]]
        return torch.einsum("efiq,eis->efqs", basis, U)

    def superbee(self, U):
        ub = torch.einsum("ei,eis->es", self.mean_w, U)
        E, nf = self.side.shape
        nb = torch.arange(E, device=U.device)[:, None].repeat(1, nf)
        nb[self.ie[:, 0], self.if_[:, 0]] = self.ie[:, 1]
        nb[self.ie[:, 1], self.if_[:, 1]] = self.ie[:, 0]
        interior = (nb != torch.arange(E, device=U.device)[:, None])[..., None]
        jump = ub[nb] - ub[:, None]
        dev = torch.einsum("efqs,q->efs", self.face_values(U), self.wf) / self.wf.sum() - ub[:, None]

        def pick(x, y, least):
            return torch.where(x * y <= 0.0, 0.0, torch.where((x.abs() < y.abs()) == least, x, y))

        allowed = pick(pick(2.0 * jump, dev, True), pick(jump, 2.0 * dev, True), False)
        theta = torch.clamp(allowed / torch.where(dev.abs() > 1e-12, dev, 1.0), 0.0, 1.0)
        limit = self.opts.tvb_constant * (self.area / self.area.sum())[:, None, None] * ub.abs().amax(0)
        quiet = (dev.abs() <= 1e-12) | ~interior | (dev.abs() <= limit)
        theta = torch.where(quiet, 1.0, theta).amin((1, 2))[:, None, None]
        return ub[:, None] + theta * (U - ub[:, None])

    def limit(self, U, fraction=1e-8, halvings=12):
        if self.opts.limiter == "none" or self.order == 0:
            return U
        if self.opts.limiter == "superbee":
            U = self.superbee(U)
        g, fl = self.g, self.flow
        rho_floor, p_floor = fraction * fl.stagnation_density, fraction * fl.total_pressure
        ub = torch.einsum("ei,eis->es", self.mean_w, U)
        rho = torch.clamp(ub[:, 0], min=rho_floor)
        e = torch.maximum(ub[:, 3], p_floor / (g - 1.0) + 0.5 * (ub[:, 1] ** 2 + ub[:, 2] ** 2) / rho)
        fix = torch.stack([rho - ub[:, 0], torch.zeros_like(e), torch.zeros_like(e), e - ub[:, 3]], -1)
        U = U + fix[:, None]
        ub = torch.einsum("ei,eis->es", self.mean_w, U)
        probes = torch.cat([torch.einsum("iq,eis->eqs", self.phi, U), self.face_values(U).reshape(U.shape[0], -1, 4)], 1)

        def pressure(V):
            return (g - 1.0) * (V[..., 3] - 0.5 * (V[..., 1] ** 2 + V[..., 2] ** 2) / torch.clamp(V[..., 0], min=1e-300))

        eps_r = torch.clamp(fraction * ub[:, 0], min=0.5 * rho_floor)
        eps_p = torch.clamp(fraction * pressure(ub), min=0.5 * p_floor)
        dev = probes - ub[:, None]

        def ok(theta):
            return pressure(ub[:, None] + theta[:, None, None] * dev).amin(1) >= eps_p

        rmin = probes[..., 0].amin(1)
        low = rmin < eps_r
        one = torch.ones_like(rmin)
        bad = low | ~ok(one)
        gap = ub[:, 0] - rmin
        top = torch.where(low, torch.clamp((ub[:, 0] - eps_r) / torch.where(gap > 0.0, gap, one), 0.0, 1.0), one)
        lo, hi, fine = torch.zeros_like(top), top, ok(top)
        for _ in range(halvings):
            mid = 0.5 * (lo + hi)
            good = ok(mid)
            lo, hi = torch.where(good, mid, lo), torch.where(good, hi, mid)
        theta = torch.where(fine, top, lo)[:, None, None]
        return torch.where(bad[:, None, None], ub[:, None] + theta * (U - ub[:, None]), U)

    def step_size(self, wave, scheme):
        limits = {"ssprk3": (1.437, 2.337, 2.240), "euler": (1.169, 1.337, 0.775)}[scheme]
        p, cfl = self.order, self.opts.cfl
        if cfl is None:
            cfl = 0.7 * (limits[p] if p < 3 else 1.32 * (2 * p + 1) / (p + 1) if scheme == "ssprk3" else 0.7)
        return cfl / (2 * p + 1) * 2.0 * self.area / torch.clamp(wave, min=self.FLOOR)

    def march(self, U, steps):
        scheme = "euler" if self.order == 0 else "ssprk3"
        at = self.flow.stagnation_sound_speed
        weight = torch.tensor([1.0, 1.0 / at, 1.0 / at, 1.0 / at ** 2], dtype=U.dtype, device=U.device)
        res = 0.0
        for _ in range(steps):
            F, wave = self.rate(U)
            dt = self.step_size(wave, scheme)[:, None, None]
            res = float(torch.sqrt(((F * weight) ** 2).mean()))
            V = self.limit(U + dt * F)
            if scheme == "ssprk3":
                V = self.limit(0.75 * U + 0.25 * (V + dt * self.rate(V)[0]))
                V = self.limit((1.0 / 3.0) * U + (2.0 / 3.0) * (V + dt * self.rate(V)[0]))
            U = V
        return U, res

    def adjoint(self, U, seed, steps):
        U = U.clone().requires_grad_(True)
        R, wave = self.residual(U)
        dt = self.step_size(wave.detach(), "ssprk3")[:, None, None]

        def defect(lam):
            return torch.autograd.grad(R, U, lam, retain_graph=True)[0] - seed

        def f(lam):
            return -torch.cholesky_solve(defect(lam), self.chol)

        lam = torch.zeros_like(seed)
        r0 = float(torch.sqrt((defect(lam) ** 2).mean()))
        for _ in range(steps):
            k0 = f(lam)
            k1 = f(lam + 0.5 * dt * k0)
            k2 = f(lam + 0.5 * dt * k1)
            k3 = f(lam + dt * k2)
            lam = lam + dt / 6.0 * (k0 + 2.0 * k1 + 2.0 * k2 + k3)
        return lam, float(torch.sqrt((defect(lam) ** 2).mean())) / r0


def _soa(U):
    return U.permute(2, 1, 0).contiguous().reshape(-1)


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        return None  # a member's march takes seconds here, and a sweep has many
    if path in ("stage", "residual"):
        ops, flow, opts, U = _residual_parts(case, seed)
        plain = _Plain(ops, flow, opts)
        if path == "residual":
            R, wave = plain.residual(U)
            return {"R": _soa(R), "wave": wave}
        U, res = plain.march(U, case["steps"])
        return {"U": _soa(U), "residual": torch.tensor([res], dtype=torch.float64)}
    cs = _nozzle(case, seed)
    plain = _Plain(cs.operators, cs.flow, cs.options)
    if path == "march":
        U, res = plain.march(torch.as_tensor(np.asarray(cs.initial_state(), float), device="cuda"), case["steps"])
        return {"U": U, "residual": res}
    U = _flow_state(case, cs)
    if path == "gradient":
        lam = _cotangent(_soa(U), seed)
        X, pb, U = (t.clone().requires_grad_(True) for t in (plain.X, plain.p_back, U))
        plain.p_back = pb
        plain.geometry(X)
        R = _soa(plain.residual(U)[0])
        gU, gX, gpb = torch.autograd.grad(R, (U, X, pb), lam)
        return {"R": R.detach(), "gU": _soa(gU), "gX": gX, "gpb": gpb}
    model = _model(cs.operators, cs.flow, cs.options)
    lam, rel = plain.adjoint(U, _thrust_seed(model, U), case["steps"])
    return {"lam": _soa(lam), "rel": rel, "iterations": None}
