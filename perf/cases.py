"""Workloads for measuring the framework: what a program that uses it has it do.

Each case is one call (or one short sequence of calls) of the public Python
interface: solves, adjoint gradients, assembly, time steps, Newton, the
multigrid as a preconditioner.  `kind` names the call, the other entries its
grid, precision and options:

  solve      x = A^{-1} b with multigrid-preconditioned CG / BiCGStab
  gradient   u(m, f), then dJ/dm and dJ/df, through torch.autograd
  assemble   new element coefficients and source: operator, right-hand side
             and the residual b - A u (what precedes every solve)
  timestep   one step of the theta scheme: prepare, assemble, solve
  newton     NewtonSolver on the assembled operator: defect, jacobian,
             multigrid set-up, linear solve
  cycle      one application of the multigrid, the preconditioner of a solver
             that the program runs itself

Grids are the unit square / cube: mx x my x mz coarse cells refined nref
times ("quad", "hex", or "tet": six Kuhn tetrahedra per cell), or with
"mesh": "free" an unstructured coarse mesh (those tetrahedra with moved
vertices) handed over as arrays and refined nref times.
"""
import collections
import math

import numpy as np
import torch

import ugcore_gb300 as ug
from ugcore_gb300 import adjoint, problems

DEVICE = "cuda"
DEFAULTS = dict(kind="solve", elem="hex", mesh="box", mx=2, my=2, mz=2, nref=3, precision="fp64", coef="one",
                flow=False, smoother="jacobi", rap=False)


def _case(name=None, **kw):
    c = dict(DEFAULTS, **kw)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the smallest solve of the benchmark problems, 129^2: launches and latency
        _case("poisson_quad_129", elem="quad", nref=6),
        # the headline: 3D Poisson on 129^3 hexahedra in FP64
        _case("poisson_hex_129", nref=6),
        # variable coefficients on Kuhn tetrahedra, FP32 multigrid in FP64 CG
        _case("lognormal_tet_129_mixed", elem="tet", mx=4, my=4, mz=4, nref=5, precision="mixed", coef="field"),
        # the largest: convection-diffusion, 193^3, BiCGStab
        _case("convection_hex_193_mixed", mx=3, my=3, mz=3, nref=6, precision="mixed", flow=True),
        # the inverse problem's gradient, 257^2, once per optimisation step
        _case("gradient_quad_257", kind="gradient", elem="quad", nref=7, coef="element"),
        # the adjoint of a flow problem, on a box with unequal sides in cells
        _case("gradient_flow_hex_mixed", kind="gradient", mx=3, my=2, mz=2, nref=5, precision="mixed",
              coef="element", flow=True),
        # re-assembly for new coefficients (every optimisation or nonlinear step)
        _case("assemble_hex_129", kind="assemble", nref=6, coef="element"),
        # the same on an unstructured mesh, 1.6 million tetrahedra
        _case("assemble_free_tet", kind="assemble", elem="tet", mesh="free", nref=5, coef="element"),
        # a solve on an unstructured mesh (general sparse operators, stored transfers)
        _case("solve_free_tet_mixed", elem="tet", mesh="free", mx=3, my=3, mz=3, nref=5, precision="mixed",
              coef="field"),
        # one Crank-Nicolson step, 97^3
        _case("timestep_hex_97_mixed", kind="timestep", mx=3, my=3, mz=3, nref=5, precision="mixed", coef="element"),
        # Newton with a fresh jacobian and multigrid, 49^3 tetrahedra
        _case("newton_tet_49", kind="newton", elem="tet", mx=3, my=3, mz=3, nref=4, coef="field"),
        # multicolour Gauss-Seidel multigrid as a preconditioner, upwind operator
        _case("cycle_gs_hex_97_mixed", kind="cycle", mx=3, my=3, mz=3, nref=5, precision="mixed", flow=True,
              smoother="mcgs"),
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "gradient", "assemble", "timestep", "newton", "cycle"])
    elem = rng.choice(["quad", "hex", "hex", "tet", "tet"])
    free = elem == "tet" and kind in ("solve", "assemble") and rng.random() < 0.4
    # cells per direction, spread over their logarithm
    lo, hi = (24, 400) if elem == "quad" else ((12, 80) if free else (12, 127))
    cells = lo * (hi / lo) ** rng.random()
    nref = max(1, int(math.log2(cells / 2)))
    m = max(2, round(cells / 2 ** nref))
    mx, my, mz = (min(4, max(2, m + rng.choice((-1, 0, 0, 1)))) for _ in range(3))
    flow = elem == "hex" and kind in ("solve", "gradient", "cycle") and rng.random() < 0.4
    coef = "element" if kind in ("gradient", "assemble") else rng.choice(["one", "field", "element"])
    if flow and kind != "gradient":
        coef = "one"
    if free and coef == "one":
        coef = "field"
    smoother = rng.choice(["jacobi", "jacobi", "mcgs", "mcsgs", "ilu"]) if kind == "cycle" else "jacobi"
    rap = kind == "solve" and not free and rng.random() < 0.2
    return _case(kind=kind, elem=elem, mesh="free" if free else "box", mx=mx, my=my, mz=mz, nref=nref,
                 precision=rng.choice(["fp64", "mixed"]), coef=coef, flow=flow, smoother=smoother, rap=rap)


# ------------------------------------------------------------------ inputs --
def _cells(case):
    s = 1 << case["nref"]
    return case["mx"] * s, case["my"] * s, (case["mz"] * s if case["elem"] != "quad" else 1)


def _dim(case):
    return 2 if case["elem"] == "quad" else 3


def _counts(case):
    """(vertices, elements) of the finest level"""
    if case["mesh"] == "free":
        return _free_counts(case)
    cx, cy, cz = _cells(case)
    nv = (cx + 1) * (cy + 1) * (cz + 1 if _dim(case) == 3 else 1)
    return nv, cx * cy * cz * (6 if case["elem"] == "tet" else 1)


def _free_counts(case):
    """by the Euler characteristic 1 of a ball: regular refinement turns
    (v, e, f, t) into (v + e, 2e + 3f + t, 4f + 8t, 8t)"""
    mx, my, mz = case["mx"], case["my"], case["mz"]
    v, t = (mx + 1) * (my + 1) * (mz + 1), 6 * mx * my * mz
    f = (4 * t + 4 * (mx * my + my * mz + mz * mx)) // 2
    e = v + f - t - 1
    for _ in range(case["nref"]):
        v, e, f, t = v + e, 2 * e + 3 * f + t, 4 * f + 8 * t, 8 * t
    return v, t


Field = collections.namedtuple("Field", "nmodes k phase amp c scale")


def _field(dim, nmodes, kmax, seed):
    """random Fourier modes: a scalar field of unit variance and (c) a
    divergence-free velocity with |v| <= 1"""
    r = np.random.RandomState(seed % (1 << 32))
    k = []
    while len(k) < nmodes:
        kappa = kmax * (2 * r.rand(dim) - 1)
        if 0 < (kappa ** 2).sum() <= kmax ** 2:
            k.append(2 * math.pi * kappa)
    k, phase = np.array(k), 2 * math.pi * r.rand(nmodes)
    c = np.cross(k, r.randn(nmodes, 3)) if dim == 3 else np.zeros((nmodes, 3))
    bound = np.sqrt((c ** 2).sum(1)).sum()
    return Field(nmodes, k, phase, math.sqrt(2.0 / nmodes), c, 1.0 / bound if bound > 0 else 1.0)


def _eval_field(field, x):
    """the scalar field at the points x (n, dim), a CUDA tensor"""
    k, phase = _cuda(field.k), _cuda(field.phase)
    g = torch.zeros(x.shape[0], dtype=torch.float64, device=x.device)
    for j in range(field.nmodes):
        g += torch.cos(x @ k[j] + phase[j])
    return field.amp * g


def _cuda(a):
    return torch.as_tensor(a, dtype=torch.float64, device=DEVICE)


def _random(n, seed, which):
    """n values U[-1, 1]"""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(1000003 * seed + which)
    return 2 * torch.rand(n, generator=g, dtype=torch.float64, device=DEVICE) - 1


DIFFUSION = 1e-2        # of the flow problems, with cell Peclet number 10
FACTOR = 2.0            # K = exp(2 g): a contrast of about 1e4
THETA, DT = 0.5, 1e-3   # Crank-Nicolson


def _coef_field(case, seed):
    return _field(_dim(case), 64 if _dim(case) == 3 else 32, 8.0, 7919 * seed + 1)


def _flow_field(case, seed):
    f = _field(3, 16, 2.0, 7919 * seed + 2)
    return f, 10.0 * 2.0 * DIFFUSION * max(_cells(case))


def _log_coef(case, seed):
    """m per element of the finest level (kind of the adjoint and assembly cases)"""
    if case["mesh"] == "free":
        return _random(_counts(case)[1], seed, 3)
    cent = _centroids(case)
    m = _eval_field(_coef_field(case, seed), cent)
    return math.log(DIFFUSION) + 0.2 * m if case["flow"] else m


def _centroids(case):
    """element centroids of a box mesh"""
    n = _cells(case)[:_dim(case)]
    axes = [torch.arange(c, dtype=torch.float64, device=DEVICE) for c in n]
    g = torch.meshgrid(*reversed(axes), indexing="ij")
    org = torch.stack([a.reshape(-1) for a in reversed(g)], 1)
    h = _cuda([1.0 / c for c in n])
    if case["elem"] != "tet":
        return (org + 0.5) * h
    off = _cuda(np.array([np.mean(t, 0) for t in _kuhn()]))
    return ((org[:, None, :] + off[None]) * h).reshape(-1, 3)


def _kuhn():
    """corner offsets of the six tetrahedra of a cell"""
    out = []
    for a, b in ((0, 1), (0, 2), (1, 0), (1, 2), (2, 0), (2, 1)):
        p = np.zeros((4, 3), int)
        p[1:, a] = 1
        p[2:, b] = 1
        p[3] = 1
        out.append(p)
    return out


def _interior(case):
    """1 at the vertices inside the domain of a box mesh, 0 on its boundary"""
    n = _cells(case)[:_dim(case)]
    t = torch.zeros([c + 1 for c in reversed(n)], dtype=torch.float64, device=DEVICE)
    t[(slice(1, -1),) * len(n)] = 1.0
    return t.reshape(-1)


def _free_coarse(case, seed):
    """the coarse unstructured mesh: a box's tetrahedra, its vertices moved
    (those of the boundary inside their faces), positively oriented"""
    m = (case["mx"], case["my"], case["mz"])
    r = np.random.RandomState((7919 * seed + 5) % (1 << 32))
    idx = np.stack(np.meshgrid(*[np.arange(c + 1) for c in m], indexing="ij"), -1)
    idx = idx.transpose(2, 1, 0, 3).reshape(-1, 3)
    x = idx / np.array(m, float)
    move = 0.2 * (r.rand(*x.shape) - 0.5) / np.array(m)
    move[(idx == 0) | (idx == np.array(m))] = 0.0
    x = x + move
    elems = []
    for k in range(m[2]):
        for j in range(m[1]):
            for i in range(m[0]):
                for t in _kuhn():
                    p = t + np.array([i, j, k])
                    e = list(p[:, 0] + (m[0] + 1) * (p[:, 1] + (m[1] + 1) * p[:, 2]))
                    if np.linalg.det(x[e[1:]] - x[e[0]]) < 0:
                        e[1], e[2] = e[2], e[1]
                    elems.append(e)
    return x, np.array(elems, np.int32)


# ----------------------------------------------------------------- prepare --
_context = None


def _ctx():
    """one context for the process, as a program keeps it"""
    global _context
    if _context is None:
        _context = ug.Context(0)
    return _context


def _hierarchy(case, seed):
    if case["mesh"] == "free":
        x, e = _free_coarse(case, seed)
        return ug.UnstructuredHierarchy.from_arrays(_ctx(), case["elem"], x, e, num_refinements=case["nref"])
    return ug.StructuredHierarchy(_ctx(), case["elem"], case["mx"], case["my"], case["mz"], case["nref"])


def _multigrid(case, disc):
    g = ug.GeometricMultiGrid(disc)
    g.set_smoother({"jacobi": ug.Jacobi(0.6), "mcgs": ug.GaussSeidel(1.0), "mcsgs": ug.SymmetricGaussSeidel(1.0),
                    "ilu": ug.ILU(1.0)}[case["smoother"]])
    g.set_num_presmooth(2)
    g.set_num_postsmooth(2)
    g.set_precision(case["precision"])
    g.set_rap(case["rap"])
    return g


def _reduction(case):
    """of the defect; the solution of a flow problem follows its defect less
    closely, and BiCGStab's last steps depend on rounding"""
    return 1e-12 if case["flow"] else 1e-10


def _krylov(case, gmg):
    s = (ug.BiCGStab if case["flow"] else ug.CG)(_ctx())
    s.set_preconditioner(gmg)
    s.set_convergence_check(ug.StdConvCheck(200, 1e-300, _reduction(case)))
    return s


def _vector(t):
    return ug.GPUVector(_ctx(), wrap=t)


def prepare(case, seed):
    if case["kind"] == "gradient":
        return _prepare_gradient(case, seed)
    st = {"case": case}
    hier = st["hier"] = _hierarchy(case, seed)
    disc = st["disc"] = ug.DomainDiscretization(hier)
    n = hier.num_vertices()
    st["f"], st["u_t"] = _random(n, seed, 1), _random(n, seed, 2)
    if case["kind"] == "timestep":
        st["u_t"] *= _interior(case)
    if case["coef"] == "element":
        st["m"] = _log_coef(case, seed)
    torch.cuda.synchronize()   # the library reads them on its own stream
    if case["coef"] == "one":
        disc.set_diffusion(DIFFUSION if case["flow"] else 1.0)
    elif case["coef"] == "field":
        disc.set_diffusion_field(_coef_field(case, seed), factor=FACTOR)
    else:
        disc.set_log_diffusion(st["m"])
    if case["flow"]:
        disc.set_velocity_field(*_flow_field(case, seed))
        disc.set_upwind("full")
    disc.set_source(st["f"])
    A = st["A"] = ug.GPUSparseMatrix(_ctx())
    for name in ("b", "x", "y"):
        st[name + "_t"] = torch.zeros(n, dtype=torch.float64, device=DEVICE)
        st[name] = _vector(st[name + "_t"])
    st["u"] = _vector(st["u_t"])
    torch.cuda.synchronize()
    if case["kind"] == "newton":
        gmg = st["gmg"] = _multigrid(case, disc)
        lin = st["solver"] = _krylov(case, gmg)
        newton = st["newton"] = ug.NewtonSolver(_ctx())
        newton.set_linear_solver(lin)
        newton.set_convergence_check(ug.StdConvCheck(10, 1e-50, 1e-8))
        newton.init(ug.AssembledOperator(disc))
        return st
    if case["kind"] == "timestep":
        td = st["td"] = ug.ThetaTimeStep(disc, THETA)
        td.prepare_step(st["u"], 0.0, DT)
        td.assemble_linear(A, st["b"])
    else:
        disc.assemble_linear(A, st["b"])
    if case["kind"] != "assemble":
        gmg = st["gmg"] = _multigrid(case, disc)
        if case["kind"] == "timestep":
            gmg.set_discretization(st["td"])
        gmg.init(A)
        if case["kind"] != "cycle":
            st["solver"] = _krylov(case, gmg)
            st["solver"].init(A)
    _ctx().synchronize()
    return st


def _prepare_gradient(case, seed):
    cfg = problems.config("", elem=case["elem"], mx=case["mx"], my=case["my"], mz=case["mz"], nref=case["nref"],
                          precision=case["precision"], solver="bicgstab" if case["flow"] else "cg",
                          rel_red=_reduction(case))
    n = _counts(case)[0]
    m, f, data = _log_coef(case, seed), _random(n, seed, 1), _random(n, seed, 2)
    torch.cuda.synchronize()
    p = adjoint.DifferentiableProblem(_ctx(), cfg, m, f)
    if case["flow"]:
        p.disc.set_velocity_field(*_flow_field(case, seed))
        p.disc.set_upwind("full")
    return {"case": case, "problem": p, "m": m.requires_grad_(), "f": f.requires_grad_(), "data": 1e-2 * data}


# --------------------------------------------------------------------- run --
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _run_solve(s):
    s["x"].set(0.0)
    s["solver"].apply(s["x"], s["b"])
    return s["x_t"]


def _run_gradient(s):
    u = adjoint.fv1_solve(s["m"], s["f"], s["problem"])
    loss = 0.5 * ((u - s["data"]) ** 2).sum()
    gm, gf = torch.autograd.grad(loss, (s["m"], s["f"]))
    return u.detach(), gm, gf


def _run_assemble(s):
    s["disc"].set_log_diffusion(s["m"])
    s["disc"].set_source(s["f"])
    s["disc"].assemble_linear(s["A"], s["b"])
    s["A"].axpy(s["y"], 1.0, s["b"], -1.0, s["u"])
    return s["b_t"], s["y_t"]


def _run_timestep(s):
    s["td"].prepare_step(s["u"], 0.0, DT)
    s["td"].assemble_linear(s["A"], s["b"])
    s["x"].set(0.0)
    s["solver"].apply(s["x"], s["b"])
    return s["b_t"], s["x_t"]


def _run_newton(s):
    s["x"].set(0.0)
    s["newton"].prepare(s["x"])
    s["newton"].apply(s["x"])
    return s["x_t"]


def _run_cycle(s):
    s["gmg"].apply(s["x"], s["u"])
    return s["x_t"]


# -------------------------------------------------------------------- work --
def work(case):
    """each input read and each output written once; a solve reads its
    operator at least once"""
    nv, ne = _counts(case)
    nnz = nv * {"quad": 9, "hex": 27, "tet": 15}[case["elem"]]
    k = {"quad": 4, "hex": 8, "tet": 4}[case["elem"]]
    assembly = 2 * ne * k * k
    b, f = {
        "solve": (8 * nnz + 16 * nv, 2 * nnz),
        "cycle": (8 * nnz + 16 * nv, 2 * nnz),
        "gradient": (16 * ne + 32 * nv, 2 * assembly + 4 * nnz),
        "assemble": (8 * ne + 32 * nv + 8 * nnz, assembly + 2 * nnz),
        "timestep": (8 * ne + 32 * nv + 8 * nnz, assembly + 2 * nnz),
        "newton": (8 * ne + 16 * nv + 8 * nnz, 2 * assembly + 2 * nnz),
    }[case["kind"]]
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact --
# The same discretisation in plain torch, FP64: box-method element matrices,
# Krylov iterations down to rounding.
def _unit_matrices(case, h):
    """per element class: corner offsets and the element matrix of K = 1"""
    dim = len(h)
    if case["elem"] == "tet":
        out = []
        for p in _kuhn():
            x = p * h
            out.append((p, _p1_stiffness(x[None])[0]))
        return out
    corners = np.array([[(q >> d) & 1 for d in range(dim)] for q in range(1 << dim)])
    A = np.zeros((len(corners), len(corners)))
    for fr, to, ip, normal in _scvfs(dim, h):
        for j, c in enumerate(corners):
            w = np.where(c == 1, ip, 1 - ip)
            grad = [(1 if c[d] else -1) / h[d] * np.prod(np.delete(w, d)) for d in range(dim)]
            flux = -np.dot(grad, normal)
            A[fr, j] += flux
            A[to, j] -= flux
    return [(corners, A)]


def _scvfs(dim, h):
    """(from, to, integration point in the unit cell, area normal) of the
    control-volume faces of a box, corners numbered by their bits"""
    out = []
    for d in range(dim):
        for q in range(1 << dim):
            if (q >> d) & 1:
                continue
            ip = np.array([0.5 if e == d else (0.75 if (q >> e) & 1 else 0.25) for e in range(dim)])
            n = np.zeros(dim)
            n[d] = np.prod([h[e] / 2 for e in range(dim) if e != d])
            out.append((q, q | (1 << d), ip, n))
    return out


def _p1_stiffness(x):
    """P1 stiffness matrices of tetrahedra x (n, 4, 3)"""
    e = x[:, 1:] - x[:, :1]
    inv = np.linalg.inv(e) if isinstance(e, np.ndarray) else torch.linalg.inv(e)
    det = abs(np.linalg.det(e)) if isinstance(e, np.ndarray) else torch.linalg.det(e).abs()
    cat = np.concatenate if isinstance(e, np.ndarray) else torch.cat
    g = cat([-inv.sum(2)[:, :, None], inv], 2)
    return (g.transpose(0, 2, 1) if isinstance(e, np.ndarray) else g.transpose(1, 2)) @ g * (det / 6)[:, None, None]


class _Box:
    """the FV1 operator of a box mesh as diagonals over its vertices"""

    def __init__(self, case, seed):
        self.case, self.dim = case, _dim(case)
        self.n = _cells(case)[:self.dim]
        self.h = np.array([1.0 / c for c in self.n])
        self.shape = [c + 1 for c in reversed(self.n)]
        self.K = self._coefficients(seed)
        self.unit = _unit_matrices(case, self.h)
        self.diag = {}
        for p, (corners, A) in enumerate(self.unit):
            for i, ci in enumerate(corners):
                for j, cj in enumerate(corners):
                    self._add(ci, cj, self.K[p] * A[i, j])
        if case["flow"]:
            self._convection(seed)
        self.inside = _interior(case)

    def _coefficients(self, seed):
        case, nc = self.case, len(_kuhn()) if self.case["elem"] == "tet" else 1
        if case["coef"] == "one":
            K = torch.full((nc,), DIFFUSION if case["flow"] else 1.0, dtype=torch.float64, device=DEVICE)
            return [k.expand(list(reversed(self.n))) for k in K]
        m = FACTOR * _eval_field(_coef_field(case, seed), _centroids(case)) if case["coef"] == "field" \
            else _log_coef(case, seed)
        return list(torch.exp(m).reshape(*reversed(self.n), nc).unbind(-1))

    def _at(self, corner):
        """the vertices that are this corner of a cell"""
        return tuple(slice(int(corner[d]), int(corner[d]) + self.n[d]) for d in reversed(range(self.dim)))

    def _add(self, ci, cj, value):
        off = tuple(int(v) for v in (cj - ci))
        if off not in self.diag:
            self.diag[off] = torch.zeros(self.shape, dtype=torch.float64, device=DEVICE)
        self.diag[off][self._at(ci)] += value

    def _convection(self, seed):
        field, scale = _flow_field(self.case, seed)
        k, c, ph = _cuda(field.k), _cuda(field.c), _cuda(field.phase)
        corners = self.unit[0][0]
        axes = [torch.arange(m, dtype=torch.float64, device=DEVICE) for m in self.n]
        g = torch.meshgrid(*reversed(axes), indexing="ij")
        for fr, to, ip, normal in _scvfs(self.dim, self.h):
            d = int(np.argmax(normal))
            x = [(g[self.dim - 1 - e] + ip[e]) * self.h[e] for e in range(self.dim)]
            v = torch.zeros_like(x[0])
            for j in range(field.nmodes):
                v -= torch.sin(sum(k[j, e] * x[e] for e in range(self.dim)) + ph[j]) * c[j, d]
            flux = scale * field.scale * normal[d] * v
            up, dn = flux.clamp(min=0), flux.clamp(max=0)
            self._add(corners[fr], corners[fr], up)
            self._add(corners[fr], corners[to], dn)
            self._add(corners[to], corners[fr], -up)
            self._add(corners[to], corners[to], -dn)

    def volumes(self):
        """control volumes"""
        v = torch.zeros(self.shape, dtype=torch.float64, device=DEVICE)
        for corners, _ in self.unit:
            for c in corners:
                v[self._at(c)] += float(np.prod(self.h)) / (len(self.unit) * len(corners))
        return v.reshape(-1)

    def _pairs(self):
        """(offset, rows, columns) as slices of the vertex array"""
        for off in self.diag:
            r = [slice(max(0, -o), self.shape[self.dim - 1 - d] - max(0, o)) for d, o in enumerate(off)]
            c = [slice(max(0, o), self.shape[self.dim - 1 - d] - max(0, -o)) for d, o in enumerate(off)]
            yield off, tuple(reversed(r)), tuple(reversed(c))

    def matvec(self, u):
        """the operator without its boundary rows"""
        u, y = u.reshape(self.shape), torch.zeros(self.shape, dtype=torch.float64, device=DEVICE)
        for off, r, c in self._pairs():
            y[r].addcmul_(self.diag[off][r], u[c])
        return y.reshape(-1) * self.inside

    def rmatvec(self, v):
        """the transposed operator on the vertices inside"""
        v, y = (v * self.inside).reshape(self.shape), torch.zeros(self.shape, dtype=torch.float64, device=DEVICE)
        for off, r, c in self._pairs():
            y[c].addcmul_(self.diag[off][r], v[r])
        return y.reshape(-1) * self.inside

    def main_diagonal(self):
        return self.diag[(0,) * self.dim].reshape(-1)

    def gradient_m(self, u, lam):
        """-K_e sum_i lam_i (A1_e u)_i per element, lam = 0 on the boundary"""
        u, lam = u.reshape(self.shape), lam.reshape(self.shape)
        out = []
        for p, (corners, A) in enumerate(self.unit):
            s = torch.zeros_like(lam[self._at(corners[0])])
            for i, ci in enumerate(corners):
                for j, cj in enumerate(corners):
                    s += A[i, j] * lam[self._at(ci)] * u[self._at(cj)]
            out.append(-self.K[p] * s)
        return torch.stack(out, -1).reshape(-1)


class _Free:
    """the FV1 operator of a refined tetrahedral mesh as a sparse matrix; on
    simplices the box method's diffusion is the P1 stiffness matrix"""

    def __init__(self, case, seed):
        x, e = _free_coarse(case, seed)
        x, e = _cuda(x), torch.as_tensor(e, device=DEVICE, dtype=torch.int64)
        for _ in range(case["nref"]):
            x, e = self._refine(x, e)
        self.x, self.n = x, x.shape[0]
        if case["coef"] == "field":
            m = FACTOR * _eval_field(_coef_field(case, seed), x[e].mean(1))
        else:
            m = _log_coef(case, seed)
        S = _p1_stiffness(x[e]) * torch.exp(m)[:, None, None]
        rows, cols = e[:, :, None].expand(-1, 4, 4).reshape(-1), e[:, None, :].expand(-1, 4, 4).reshape(-1)
        A = torch.sparse_coo_tensor(torch.stack([rows, cols]), S.reshape(-1), (self.n, self.n)).coalesce()
        ij = A.indices()
        self.diagonal = torch.zeros(self.n, dtype=torch.float64, device=DEVICE)
        on = ij[0] == ij[1]
        self.diagonal[ij[0][on]] = A.values()[on]
        self.A = A.to_sparse_csr()
        vol = torch.linalg.det(x[e][:, 1:] - x[e][:, :1]).abs() / 24
        self.vol = torch.zeros(self.n, dtype=torch.float64, device=DEVICE)
        self.vol.index_add_(0, e.reshape(-1), vol[:, None].expand(-1, 4).reshape(-1))
        self.inside = ((x > 0) & (x < 1)).all(1).double()

    @staticmethod
    def _refine(x, e):
        """vertices: the old ones, then the edge midpoints by (smaller, larger)
        end; children: four corners, then the octahedron around its shortest
        diagonal, all positively oriented"""
        n = x.shape[0]
        ends = torch.tensor([[0, 1], [1, 2], [0, 2], [0, 3], [1, 3], [2, 3]], device=DEVICE)
        a, b = e[:, ends[:, 0]], e[:, ends[:, 1]]
        key, inv = torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b), return_inverse=True)
        x = torch.cat([x, (x[key // n] + x[key % n]) * 0.5])
        m01, m12, m02, m03, m13, m23 = (n + inv).unbind(1)
        v0, v1, v2, v3 = e.unbind(1)
        diag = [(m01, m23), (m12, m03), (m02, m13)]
        ring = [(m12, m13, m03, m02), (m01, m13, m23, m02), (m01, m12, m23, m03)]
        d2 = [((x[p] - x[q]) ** 2).unbind(1) for p, q in diag]
        d2 = [(a + b) + c for a, b, c in d2]   # ties go to the first
        best = torch.where((d2[1] < d2[0]) & ~(d2[2] < d2[1]), 1, torch.where(d2[2] < torch.minimum(d2[0], d2[1]), 2, 0))

        def pick(options):
            return torch.stack(options, 1).gather(1, best[:, None])[:, 0]

        d0, d1 = pick([d[0] for d in diag]), pick([d[1] for d in diag])
        r = [pick([q[j] for q in ring]) for j in range(4)]
        ch = [(v0, m01, m02, m03), (m01, v1, m12, m13), (m02, m12, v2, m23), (m03, m13, m23, v3)]
        ch += [(d0, d1, r[j], r[(j + 1) % 4]) for j in range(4)]
        e = torch.stack([torch.stack(c, 1) for c in ch], 1).reshape(-1, 4)
        turned = torch.linalg.det(x[e][:, 1:] - x[e][:, :1]) < 0
        return x, torch.where(turned[:, None], e[:, [0, 2, 1, 3]], e)

    def volumes(self):
        return self.vol

    def matvec(self, u):
        return (self.A @ u) * self.inside

    def main_diagonal(self):
        return self.diagonal


def _cg(apply, diag, b, most=20000):
    """Jacobi-preconditioned CG down to rounding"""
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rz, stop = z.clone(), torch.dot(r, z), 1e-15 * float(torch.linalg.norm(b))
    for it in range(most):
        q = apply(p)
        alpha = rz / torch.dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 20 == 0 and float(torch.linalg.norm(r)) <= stop:
            break
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


def _bicgstab(apply, diag, b, most=20000):
    """Jacobi-preconditioned BiCGStab, restarted from the true residual"""
    x, stop = torch.zeros_like(b), 1e-13 * float(torch.linalg.norm(b))
    for _ in range(6):
        r = b - apply(x)
        if float(torch.linalg.norm(r)) <= stop:
            break
        r0, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
        rho = alpha = omega = torch.ones((), dtype=torch.float64, device=DEVICE)
        for it in range(most):
            new = torch.dot(r0, r)
            p = r + (new / rho) * (alpha / omega) * (p - omega * v)
            rho = new
            ph = p / diag
            v = apply(ph)
            alpha = rho / torch.dot(r0, v)
            s = r - alpha * v
            sh = s / diag
            t = apply(sh)
            omega = torch.dot(t, s) / torch.dot(t, t)
            x += alpha * ph + omega * sh
            r = s - omega * t
            if it % 10 == 0 and not float(torch.linalg.norm(r)) > stop:
                break
    return x


def exact(case, seed):
    if case["kind"] == "cycle":
        return None
    op = _Free(case, seed) if case["mesh"] == "free" else _Box(case, seed)
    n = op.inside.numel()
    vol, inside = op.volumes(), op.inside
    f, u = _random(n, seed, 1), _random(n, seed, 2)
    b = f * vol * inside
    diag = torch.where(inside > 0, op.main_diagonal(), torch.ones_like(inside))

    def solve(apply, rhs):
        return (_bicgstab if case["flow"] else _cg)(apply, diag, rhs)

    if case["kind"] in ("solve", "newton"):
        return solve(op.matvec, b)
    if case["kind"] == "assemble":
        return b, b - op.matvec(u) - (1 - inside) * u
    if case["kind"] == "timestep":
        u = u * inside
        rhs = (vol * u - (1 - THETA) * DT * op.matvec(u) + DT * vol * f) * inside
        diag = torch.where(inside > 0, vol + THETA * DT * op.main_diagonal(), torch.ones_like(inside))
        return rhs, solve(lambda v: vol * v * inside + THETA * DT * op.matvec(v), rhs)
    x = solve(op.matvec, b)
    lam = solve(op.rmatvec, (x - 1e-2 * u) * inside)
    return x, op.gradient_m(x, lam), lam * vol * inside
