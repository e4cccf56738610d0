"""Performance cases of the forward-solve path, measured through the public Python API.

A case is one call (or the short chain of calls) that a modelling or inversion
program makes over and over: applying the operator, assembling it, building
and applying the preconditioner, solving one right-hand side the way the
reference does, solving blocks of right-hand sides on the batched path,
estimating errors, reading receiver fields, predicting initial guesses.
Meshes come from the package's own generator at the sizes of its test and
benchmark configurations (MT halfspaces with topography and anisotropic
bodies, marine CSEM); resistivities, frequencies, sources, receivers and
vectors come from the seed.

listed() and draw() give cases, prepare() the state a program holds before
the call, run() one pass, work() the bytes and operations a pass cannot do
without, exact() the outputs in plain 64-bit torch where they have a value
that does not depend on the method.
"""

import functools
import math

import numpy as np
import torch

import emfem_b200 as E
from emfem_b200 import meshgen as mg

PI = math.pi
MU = 4 * PI * 1e-7
DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one application of the complex operator on a coarse mesh: a caller's
        # own Krylov loop or a residual check in a test; latency counts
        {"name": "operator-small", "kind": "operator", "model": "mt", "tets": 4000, "k": 1},
        # the same on a production MT mesh for 8 frequencies x 2 polarisations
        {"name": "operator-large", "kind": "operator", "model": "mt", "tets": 1500000, "k": 16},
        # a new conductivity model in an inversion: assembly, then the
        # operator on both polarisations
        {"name": "assemble", "kind": "assemble", "model": "mt", "tets": 600000, "k": 2},
        # goal-oriented error indicators of an MT run (two primal solutions
        # and the dual one), and of a CSEM run into the caller's own buffers
        {"name": "estimate-mt", "kind": "estimate", "model": "mt", "tets": 300000},
        {"name": "estimate-csem", "kind": "estimate_dev", "model": "csem", "tets": 80000},
        # fields of a solved block at a 21 x 21 receiver grid
        {"name": "fields", "kind": "fields", "model": "mt", "tets": 100000, "k": 16, "receivers": 441},
        # initial guesses for the next frequencies of a sweep: quadratic
        # interpolation in log f over 16 solved columns of two sources
        {"name": "guess", "kind": "guess", "model": "mt", "tets": 200000, "k": 16, "targets": 16, "network": 3},
        # one application of the reference-facing preconditioner (two FCG
        # solves with the FP64 AMS of one frequency) for a caller's own Krylov loop
        {"name": "precondition", "kind": "precondition", "model": "mt", "tets": 50000},
        # the drop-in's whole per-frequency step: assembly, preconditioner,
        # one CSEM right-hand side solved in FP64
        {"name": "solve-single", "kind": "single", "model": "csem", "tets": 10000},
        # a small batched forward run: 3 frequencies x 2 transmitters
        {"name": "forward-small", "kind": "forward", "model": "csem", "tets": 5000, "freqs": 3, "sources": 2},
        # the full-size marine CSEM configuration: 3 frequencies, one transmitter
        {"name": "forward-csem", "kind": "forward", "model": "csem", "tets": 80000, "freqs": 3, "sources": 1},
        # MT with topography: 8 frequencies x 2 polarisations on a mesh kept
        # to a pass of about a second; the package's headline workload
        {"name": "forward-mt", "kind": "forward", "model": "mt", "tets": 120000, "freqs": 8, "sources": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operator", "operator", "assemble", "estimate", "estimate_dev", "fields", "guess",
                       "precondition", "single", "forward", "forward", "forward"])
    model = rng.choice(["mt", "csem"])
    c = {"kind": kind, "model": model}
    if kind == "operator":
        c.update(tets=_log_int(rng, 4000, 590000), k=rng.choice([1, 2, 4, 8, 16]))
    elif kind == "assemble":
        c.update(tets=_log_int(rng, 4000, 590000), k=rng.choice([1, 2]))
    elif kind == "estimate":
        c.update(tets=_log_int(rng, 4000, 290000))
    elif kind == "estimate_dev":
        c.update(tets=_log_int(rng, 4000, 79000))
    elif kind == "fields":
        c.update(tets=_log_int(rng, 4000, 99000), k=rng.choice([1, 2, 3, 8, 16]), receivers=_log_int(rng, 5, 440))
    elif kind == "guess":
        c.update(tets=_log_int(rng, 4000, 190000), k=rng.choice([6, 8, 16]), targets=rng.choice([3, 8, 16]),
                 network=rng.choice([1, 3]))
    elif kind == "precondition":
        c.update(tets=_log_int(rng, 4000, 49000))
    elif kind == "single":
        c.update(model="csem", tets=_log_int(rng, 4000, 10000))
    elif model == "csem":
        c.update(tets=_log_int(rng, 4000, 79000), freqs=rng.choice([1, 2, 3]), sources=rng.choice([1, 2, 3, 4]))
    else:
        c.update(tets=_log_int(rng, 4000, 100000), freqs=rng.choice([1, 2, 3, 4, 6, 8]), sources=2)
    return c


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _problem(model, tets):
    """Mesh, regions and survey geometry; the seed varies only what is on them."""
    if model == "mt":
        return mg.mt_halfspace_block(tets, with_block=False, topo_height=1e3, topo_sigma=5e3, n_bodies=5, seed=2)
    return mg.marine_csem(tets, n_reservoirs=1, n_tx=4, seed=3)


def _model(prob, rng):
    """Resistivities within a factor of two of the base model; air stays air."""
    rho = prob.model.rho.copy()
    ncol = 3 if prob.model.aniso_form == mg.ARBITRARY else rho.shape[1]
    first = 1 if prob.survey.kind == "mt" else 2  # the sea's resistivity is known
    rho[first:, :ncol] *= 10 ** rng.uniform(-0.3, 0.3, size=(rho.shape[0] - first, 1))
    return mg.Model(prob.model.aniso_form, rho)


def _freqs(case, rng):
    if case["model"] == "mt":
        n = case.get("freqs", 8)
        f = np.logspace(-1, 1.5, n) if n > 1 else np.array([1.0])
    else:
        f = np.array([0.25, 0.75, 1.25])[:case.get("freqs", 3)]
    return f * 10 ** rng.uniform(-0.05, 0.05, size=f.size)


def _points_in(mesh, cells, rng):
    """One point well inside each of the given cells."""
    lam = 0.1 + rng.dirichlet(np.ones(4), size=len(cells)) * 0.6
    return np.einsum("ij,ijk->ik", lam, mesh.points[mesh.tets[cells]])


def _edge_field(mesh, cols, rng):
    """A smooth complex vector field with a little roughness as edge values (n_edges, cols)."""
    p = torch.from_numpy(mesh.points).to(DEV)
    e = torch.from_numpy(mesh.edges.astype(np.int64)).to(DEV)
    t = p[e[:, 1]] - p[e[:, 0]]
    mid = (p[e[:, 1]] + p[e[:, 0]]) / 2e4
    out = torch.zeros((mesh.n_edges, cols), dtype=torch.complex128, device=DEV)
    g = torch.Generator(device=DEV).manual_seed(int(rng.integers(1 << 31)))
    noise = torch.rand((mesh.n_edges,), generator=g, dtype=torch.float64, device=DEV) * 0.02 + 1
    for j in range(cols):
        k, ph, d = (torch.from_numpy(rng.uniform(-1, 1, size=(2, 3))).to(DEV), rng.uniform(0, 6, size=2),
                    torch.from_numpy(rng.uniform(-1, 1, size=(2, 3))).to(DEV))
        for i, z in ((0, 1.0), (1, 1j)):
            out[:, j] += z * (t @ d[i]) * (torch.exp(-mid.abs().sum(1) / 4) + 0.1) * torch.cos(mid @ k[i] + ph[i])
        out[:, j] *= noise
    return out


def _earth_cells(prob, rng, n):
    """Random cells in the central part of the survey, outside the air."""
    m = prob.mesh
    cen = m.points[m.tets].mean(axis=1)
    near = np.nonzero((np.abs(cen[:, 0]) < 8e3) & (np.abs(cen[:, 1]) < 4e3) & (cen[:, 2] > 0) & (cen[:, 2] < 3e3))[0]
    return rng.choice(near, size=n, replace=n > near.size).astype(np.int32)


def _inputs(case, seed):
    """Everything a case is made of, on the host (exact() starts here too)."""
    rng = np.random.default_rng(seed)
    prob = _problem(case["model"], case["tets"])
    s = {"prob": prob, "model": _model(prob, rng), "freqs": _freqs(case, rng), "kind": case["kind"]}
    kind = case["kind"]
    if kind == "operator":
        f = np.repeat(s["freqs"], -(-case["k"] // s["freqs"].size))[:case["k"]]
        s["omegas"] = 2 * PI * f
        s["x"] = _edge_field(prob.mesh, case["k"], rng)
    elif kind == "assemble":
        s["x"] = _edge_field(prob.mesh, case["k"], rng)
    elif kind in ("estimate", "estimate_dev"):
        s["sol"] = _edge_field(prob.mesh, 3 if case["model"] == "mt" else 2, rng)
    elif kind == "fields":
        s["cells"] = _earth_cells(prob, rng, case["receivers"])
        s["rx"] = _points_in(prob.mesh, s["cells"], rng)
        s["colf"] = np.resize(s["freqs"], case["k"])
        s["x"] = _edge_field(prob.mesh, case["k"], rng)
    elif kind == "guess":
        # two sources: even columns the first, odd the second; targets lie
        # between the solved frequencies
        k, kt = case["k"], case["targets"]
        f = np.logspace(-1, 1.5, (k + 1) // 2) * 10 ** rng.uniform(-0.02, 0.02)
        s["colf"], s["src"] = np.repeat(f, 2)[:k], np.arange(k, dtype=np.int32) % 2
        tf = 10 ** rng.uniform(-0.7, 1.1, size=kt)
        s["tf"], s["tsrc"] = tf, np.arange(kt, dtype=np.int32) % 2
        s["x"] = _edge_field(prob.mesh, k, rng)
        s["seed"] = int(rng.integers(1 << 31))
    elif kind == "precondition":
        s["b"] = _edge_field(prob.mesh, 1, rng)
    elif kind == "single" or case["model"] == "csem":
        n = case.get("sources", 1)
        s["cells"] = _earth_cells(prob, rng, n)
        pos = _points_in(prob.mesh, s["cells"], rng)
        # horizontal electric dipoles of unit moment
        s["tx"] = np.concatenate([pos, rng.uniform(-30, 30, size=(n, 1)), np.zeros((n, 1)), np.ones((n, 1)),
                                  np.zeros((n, 1))], axis=1)
    return s


def _context(s, tidx):
    ctx = E.EMContext(0)
    ctx.set_mesh(s["prob"].mesh)
    ctx.set_model(s["model"])
    ctx.set_frequencies(s["freqs"])
    ctx.create_linear_system(tidx)
    return ctx


def prepare(case, seed):
    s = _inputs(case, seed)
    kind, mt = case["kind"], case["model"] == "mt"
    m = s["prob"].mesh
    ctx = s["ctx"] = _context(s, -1 if mt else 0)
    if kind == "operator":
        ctx.assemble_matrix(0)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "assemble":
        s["y"] = torch.empty_like(s["x"])
        s["omegas"] = np.full(case["k"], 2 * PI * s["freqs"][0])
    elif kind in ("estimate", "estimate_dev"):
        for j, slot in enumerate((E.XY_POLAR, E.YX_POLAR, E.SOL_DUAL) if mt else (E.SOL_CSEM, E.SOL_DUAL)):
            z = s["sol"][:, j].cpu().numpy()
            ctx.set_solution(slot, z.real, z.imag)
        n = s["sol"].shape[1]
        s["err"] = torch.empty((n - 1, m.n_tets), dtype=torch.float64, device=DEV)
        s["eta"] = torch.empty((n, m.n_tets), dtype=torch.float64, device=DEV)
    elif kind == "guess":
        s["guess"] = torch.empty((m.n_edges, case["targets"]), dtype=torch.complex128, device=DEV)
        s["network"] = case["network"]
        if s["network"] == 1:
            n = ctx.warm_start_params().size
            ctx.warm_start_params(np.random.default_rng(s["seed"]).normal(0, 0.05, size=n))
    elif kind == "precondition":
        ctx.assemble_matrix(0)
        ctx.create_pc()
        z = s["b"][:, 0].cpu().numpy()
        s["host_b"] = np.concatenate([z.real, z.imag])
    elif kind in ("single", "forward"):
        if mt:
            ctx.set_background(*mg.background_model(m, s["model"]))
            s["modes"] = np.tile([E.XY_POLAR, E.YX_POLAR], s["freqs"].size).astype(np.int32)
            s["colf"] = np.repeat(s["freqs"], 2)
        else:
            n = s["tx"].shape[0]
            s["colf"], s["cols_tx"] = np.repeat(s["freqs"], n), np.tile(s["tx"], (s["freqs"].size, 1))
        if kind == "forward":
            k = s["colf"].size
            s["rhs"] = torch.empty((m.n_edges, k), dtype=torch.complex128, device=DEV)
            s["x"] = torch.empty((m.n_edges, k), dtype=torch.complex128, device=DEV)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "operator":
        ctx.spmv_complex_dev(s["omegas"], s["x"].data_ptr(), s["y"].data_ptr())
        ctx.synchronize()
        return s["y"]
    if kind == "assemble":
        ctx.assemble_matrix(0)
        ctx.spmv_complex_dev(s["omegas"], s["x"].data_ptr(), s["y"].data_ptr())
        ctx.synchronize()
        return s["y"]
    if kind == "estimate":
        return ctx.estimate_error(0, -1 if s["sol"].shape[1] == 3 else 0)
    if kind == "estimate_dev":
        ctx.estimate_error_noalloc_dev(0, -1 if s["sol"].shape[1] == 3 else 0, s["err"].data_ptr(),
                                       s["eta"].data_ptr())
        return s["err"], s["eta"]
    if kind == "fields":
        return ctx.interpolate_fields_block_dev(s["colf"], s["x"].data_ptr(), s["rx"], s["cells"])
    if kind == "guess":
        ctx.warm_start_predict(s["colf"], s["src"], s["x"].data_ptr(), s["tf"], s["tsrc"], s["guess"].data_ptr(),
                               network=s["network"])
        return s["guess"]
    if kind == "precondition":
        return ctx.pc_apply_b(s["host_b"])
    ctx.assemble_matrix(0)
    if kind == "single":
        ctx.create_pc()
        sr, si = ctx.assemble_rhs_csem(0, s["tx"][0], s["cells"][:1])
        ctx.solve_linear_system(E.SOL_CSEM, sr, si)
        return ctx.get_solution(E.SOL_CSEM)
    if "modes" in s:
        ctx.assemble_rhs_mt_block_dev(s["colf"], s["modes"], s["rhs"].data_ptr())
    else:
        ctx.assemble_rhs_csem_block_dev(s["colf"], s["cols_tx"], s["rhs"].data_ptr())
    ctx.solve_block_dev(s["colf"], s["rhs"].data_ptr(), s["x"].data_ptr(), rtol=1e-8, max_it=200)
    return s["x"]


# ---------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once.  Solves count the mesh, the
    operator, the right-hand sides and the solutions once each: the least any
    method moves, however many iterations it takes."""
    m = _problem(case["model"], case["tets"]).mesh
    nt, ne, nv = m.n_tets, m.n_edges, m.n_vertices
    interior = int((m.neighbors >= 0).sum()) // 2
    # edges pair up within a tet (15 pairs) and within a face two tets share (3)
    nnz = ne + 2 * (15 * nt - 3 * interior)
    kind, k = case["kind"], case.get("k", 1)
    mesh = nt * 44.0 + nv * 24.0       # vertices, edges and attribute of each tet; coordinates
    matrix = nnz * 20.0 + ne * 4.0     # column index and two values per nonzero
    if kind == "operator":
        return {"bytes": matrix + ne * k * 32.0, "flops": nnz * k * 10.0}
    if kind == "assemble":
        return {"bytes": mesh + matrix + ne * k * 32.0, "flops": nt * 1200.0 + nnz * k * 10.0}
    if kind in ("estimate", "estimate_dev"):
        n = 3 if case["model"] == "mt" else 2
        return {"bytes": mesh + nt * 32.0 + ne * n * 16.0 + nt * (2 * n - 1) * 8.0, "flops": nt * n * 2500.0}
    if kind == "fields":
        return {"bytes": case["receivers"] * (28.0 + 40 + 96 + k * (6 * 16 + 96)), "flops": case["receivers"] * k * 250.0}
    if kind == "guess":
        return {"bytes": ne * (k + case["targets"]) * 16.0, "flops": ne * case["targets"] * 12.0}
    if kind == "precondition":
        return {"bytes": matrix + ne * 32.0, "flops": nnz * 4.0}
    cols = 1 if kind == "single" else case["freqs"] * case["sources"]
    return {"bytes": mesh + matrix + ne * cols * 32.0, "flops": nt * 1200.0 + nnz * cols * 10.0}


# ---------------------------------------------------------------------------
# the outputs in plain 64-bit torch
# ---------------------------------------------------------------------------
LOCAL = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


def _sigma(model):
    r = model.rho
    out = np.zeros((r.shape[0], 3, 3))
    for i, row in enumerate(r):
        if model.aniso_form == mg.ISOTROPIC:
            out[i] = np.eye(3) / row[0]
        elif model.aniso_form == mg.VERTICAL:
            out[i] = np.diag([1 / row[0], 1 / row[0], 1 / row[1]])
        else:
            a, b, c = np.deg2rad(row[3:6])
            x = np.array([[1, 0, 0], [0, np.cos(a), np.sin(a)], [0, -np.sin(a), np.cos(a)]])
            y = np.array([[np.cos(b), 0, -np.sin(b)], [0, 1, 0], [np.sin(b), 0, np.cos(b)]])
            z = np.array([[np.cos(c), np.sin(c), 0], [-np.sin(c), np.cos(c), 0], [0, 0, 1]])
            q = z @ y @ x
            out[i] = q @ np.diag(1 / row[:3]) @ q.T
    return torch.from_numpy(out).to(DEV)


class _Geometry:
    """Barycentric gradients, volumes and edge orientations of (some of) the cells."""

    def __init__(self, mesh, cells=None):
        sel = np.arange(mesh.n_tets) if cells is None else np.asarray(cells)
        self.tets = torch.from_numpy(mesh.tets[sel].astype(np.int64)).to(DEV)
        self.t2e = torch.from_numpy(mesh.tet2edge[sel].astype(np.int64)).to(DEV)
        self.edges = torch.from_numpy(mesh.edges.astype(np.int64)).to(DEV)
        self.x = torch.from_numpy(mesh.points).to(DEV)[self.tets]                     # (T, 4, 3)
        self.attr = torch.from_numpy(mesh.attr[sel].astype(np.int64)).to(DEV)
        e = self.x[:, 1:] - self.x[:, :1]
        c = torch.stack([torch.linalg.cross(e[:, 1], e[:, 2]), torch.linalg.cross(e[:, 2], e[:, 0]),
                         torch.linalg.cross(e[:, 0], e[:, 1])], 1)
        det = (e[:, 0] * c[:, 0]).sum(1)
        g = c / det[:, None, None]
        self.gr = torch.cat([-g.sum(1, keepdim=True), g], 1)                          # (T, 4, 3)
        self.vol = det / 6
        # local vertices at the ends of each local edge, lower global id first
        ab = self.edges[self.t2e]                                                     # (T, 6, 2)
        self.a = (self.tets[:, None, :] == ab[:, :, :1]).long().argmax(2)
        self.b = (self.tets[:, None, :] == ab[:, :, 1:]).long().argmax(2)
        pick = lambda i: torch.gather(self.gr, 1, i[:, :, None].expand(-1, -1, 3))    # noqa: E731
        self.ga, self.gb = pick(self.a), pick(self.b)
        self.curl = 2 * torch.linalg.cross(self.ga, self.gb)                          # (T, 6, 3)

    def basis(self, lam):
        """(T, 6, 3) edge functions at one barycentric point (T, 4) per cell."""
        return torch.gather(lam, 1, self.a)[:, :, None] * self.gb - torch.gather(lam, 1, self.b)[:, :, None] * self.ga

    def barycentric(self, y):
        return 1 + ((y[:, None] - self.x) * self.gr).sum(2)


def _element_matrices(mesh, model):
    """(geometry, C, Ms) with the Dirichlet rows and columns cleared."""
    g = _Geometry(mesh)
    s = _sigma(model)[g.attr]
    S = torch.einsum("tid,tde,tje->tij", g.gr, s, g.gr)
    C = torch.einsum("tkd,tld->tkl", g.curl, g.curl) * (g.vol / MU)[:, None, None]

    def part(p, q):  # integral of lambda_p lambda_q times the product of the other two gradients
        same = 1.0 + (p[0][:, :, None] == q[0][:, None, :]).double()
        other = S.reshape(-1, 16).gather(1, (p[1][:, :, None] * 4 + q[1][:, None, :]).reshape(-1, 36)).reshape(-1, 6, 6)
        return same * other

    ab, ba = (g.a, g.b), (g.b, g.a)
    M = (part(ab, ab) - part(ab, ba) - part(ba, ab) + part(ba, ba)) * (g.vol / 20)[:, None, None]
    bd = torch.from_numpy(mesh.edge_bdr.astype(bool)).to(DEV)[g.t2e]
    cut = bd[:, :, None] | bd[:, None, :]
    eye = torch.eye(6, dtype=torch.bool, device=DEV)
    return g, C.masked_fill(cut & ~eye, 0.0), M.masked_fill(cut, 0.0)


def _apply(g, K, x):
    """y = sum over cells of K_t x_t for complex columns."""
    y = torch.zeros_like(x)
    for j in range(x.shape[1]):
        for z in (0, 1):
            v = torch.view_as_real(x)[:, j, z][g.t2e]
            torch.view_as_real(y)[:, j, z].index_add_(0, g.t2e.reshape(-1), torch.einsum("tkl,tl->tk", K, v).reshape(-1))
    return y


def _exact_estimate(s, sol):
    mesh = s["prob"].mesh
    g = _Geometry(mesh)
    sg = _sigma(s["model"])[g.attr]
    nt = mesh.n_tets
    w = 2 * PI * float(s["freqs"][0])
    d = lambda i, j: (g.x[:, i] - g.x[:, j]).norm(dim=1)                              # noqa: E731
    la, lb, lc = d(1, 2) * d(0, 3), d(0, 2) * d(1, 3), d(0, 1) * d(2, 3)
    sh = (la + lb + lc) / 2
    rad = (sh * (sh - la) * (sh - lb) * (sh - lc)).sqrt() / (6 * g.vol)
    A, B = 0.585410196624969, 0.138196601125011
    nbr = torch.from_numpy(mesh.neighbors.astype(np.int64)).to(DEV)
    own, face = torch.nonzero(nbr > torch.arange(nt, device=DEV)[:, None], as_tuple=True)
    other = nbr[own, face]
    gp = g.gr[own, face]
    gl = gp.norm(dim=1)
    nrm = -gp / gl[:, None]
    jxw = gl * (6 * g.vol[own]).abs()
    fv = torch.tensor([[1, 2, 3], [2, 3, 0], [3, 0, 1], [0, 1, 2]], device=DEV)[face]  # (F, 3)
    fx = torch.gather(g.x[own], 1, fv[:, :, None].expand(-1, -1, 3))
    ea, eb, ec = [(fx[:, i] - fx[:, j]).norm(dim=1) for i, j in ((0, 1), (1, 2), (2, 0))]
    area = 0.25 * ((ea + eb + ec) * (eb + ec - ea) * (ec + ea - eb) * (ea + eb - ec)).sqrt()
    fd = ea * eb * ec / (4 * area)

    def field(cells, lam, u):
        """e at barycentric points lam (N, 4) of the given cells"""
        wa = torch.gather(lam, 1, g.a[cells])[:, :, None] * g.gb[cells]
        wb = torch.gather(lam, 1, g.b[cells])[:, :, None] * g.ga[cells]
        return torch.einsum("tk,tkd->td", u[g.t2e[cells]], (wa - wb).to(u.dtype))

    every = torch.arange(nt, device=DEV)
    etas = []
    for j in range(sol.shape[1]):
        u = sol[:, j]
        vol = torch.zeros(nt, dtype=torch.float64, device=DEV)
        for q in range(4):
            lam = torch.full((nt, 4), B, dtype=torch.float64, device=DEV)
            lam[:, q] = A
            vol += (torch.einsum("tde,te->td", sg.to(u.dtype), field(every, lam, u)).abs() ** 2).sum(1)
        eta = vol * w * w * g.vol / 4 * rad ** 2
        curl = torch.einsum("tk,tkd->td", u[g.t2e], g.curl.to(u.dtype))
        jump = torch.linalg.cross(curl[own] - curl[other], nrm.to(u.dtype))
        v = 3 * (jump.abs() ** 2).sum(1) * jxw
        for q in range(3):
            lam = torch.full((own.numel(), 4), 1 / 6, dtype=torch.float64, device=DEV)
            lam.scatter_(1, face[:, None], 0.0)
            lam.scatter_(1, fv[:, q:q + 1], 2 / 3)
            y = (lam[:, :, None] * g.x[own]).sum(1)
            lam2 = 1 + ((y[:, None] - g.x[other]) * g.gr[other]).sum(2)
            jd = (torch.einsum("tde,te->td", sg[own].to(u.dtype), field(own, lam, u)) -
                  torch.einsum("tde,te->td", sg[other].to(u.dtype), field(other, lam2, u)))
            v += (jd * nrm).sum(1).abs() ** 2 * jxw
        v *= fd / 2
        eta.index_add_(0, own, v)
        eta.index_add_(0, other, v)
        etas.append(eta)
    eta = torch.stack(etas)
    return (eta[:-1] * eta[-1:]).sqrt(), eta


def _exact_solve(s):
    """Dense LU of C + i w Ms per frequency, then the weak divergence condition
    G^T (b - A x) = 0, which the LU alone leaves to rounding in the air."""
    mesh = s["prob"].mesh
    g, C, M = _element_matrices(mesh, s["model"])
    n, nv = mesh.n_edges, mesh.n_vertices
    idx = (g.t2e[:, :, None] * n + g.t2e[:, None, :]).reshape(-1)
    dense = lambda K: torch.zeros(n * n, dtype=torch.float64, device=DEV).index_add_(0, idx, K.reshape(-1)).reshape(n, n)  # noqa: E731
    Cd, Md = dense(C), dense(M)
    G = torch.zeros((n, nv), dtype=torch.float64, device=DEV)
    rows = torch.arange(n, device=DEV)
    G[rows, g.edges[:, 0]], G[rows, g.edges[:, 1]] = -1.0, 1.0
    G = G[:, torch.from_numpy(mesh.vertex_bdr == 0).to(DEV)]
    MG = Md @ G
    N = G.T @ MG
    dia = N.diagonal().rsqrt()
    Nf = torch.linalg.cholesky(N * dia[:, None] * dia[None, :])
    tx, cells = s["tx"], s["cells"]
    gt = _Geometry(mesh, cells)
    phi = gt.basis(gt.barycentric(torch.from_numpy(tx[:, :3].copy()).to(DEV)))
    az, dip = np.deg2rad(tx[:, 3]), np.deg2rad(tx[:, 4])
    d = torch.from_numpy(np.stack([np.cos(az) * np.cos(dip), np.sin(az) * np.cos(dip), np.sin(dip)], 1)).to(DEV)
    src = torch.zeros((n, tx.shape[0]), dtype=torch.float64, device=DEV)
    for i in range(tx.shape[0]):
        src[gt.t2e[i], i] = (phi[i] @ d[i]) * float(tx[i, 5])
    out = []
    for f in s["freqs"] if s["kind"] == "forward" else s["freqs"][:1]:
        w = 2 * PI * float(f)
        lu = torch.linalg.lu_factor(torch.complex(Cd, w * Md))
        b = torch.complex(torch.zeros_like(src), -w * src)
        x = torch.zeros_like(b)
        for _ in range(3):
            r = b - torch.complex(Cd @ x.real - w * (Md @ x.imag), Cd @ x.imag + w * (Md @ x.real))
            x = x + torch.linalg.lu_solve(*lu, r)
            # C G = 0, so G^T (b - A x) = G^T b - i w (Ms G)^T x
            t = (G.T.to(b.dtype) @ b - 1j * w * (MG.T.to(b.dtype) @ x)) / (1j * w)
            z = torch.cholesky_solve(torch.cat([t.real, t.imag], 1) * dia[:, None], Nf) * dia[:, None]
            x = x + (G @ z[:, :t.shape[1]]) + 1j * (G @ z[:, t.shape[1]:])
        out.append(x)
    return torch.cat(out, 1)


def exact(case, seed):
    s = _inputs(case, seed)
    kind, mesh = case["kind"], s["prob"].mesh
    if kind == "operator" or kind == "assemble":
        g, C, M = _element_matrices(mesh, s["model"])
        w = s.get("omegas", np.full(case["k"], 2 * PI * s["freqs"][0]))
        return _apply(g, C, s["x"]) + 1j * torch.from_numpy(w).to(DEV) * _apply(g, M, s["x"])
    if kind in ("estimate", "estimate_dev"):
        return _exact_estimate(s, s["sol"])
    if kind == "fields":
        g = _Geometry(mesh, s["cells"])
        phi = g.basis(g.barycentric(torch.from_numpy(s["rx"]).to(DEV))).to(torch.complex128)
        u = s["x"][g.t2e]                                                             # (R, 6, k)
        w = torch.from_numpy(2 * PI * s["colf"]).to(DEV)
        e = torch.einsum("rkc,rkd->rcd", u, phi)
        h = torch.einsum("rkc,rkd->rcd", u, g.curl.to(torch.complex128)) * (1j / (w * MU))[None, :, None]
        return e, h
    if kind == "guess" and case["network"] == 3:
        out = torch.zeros((mesh.n_edges, case["targets"]), dtype=torch.complex128, device=DEV)
        for j, (f, src) in enumerate(zip(s["tf"], s["tsrc"])):
            c = np.nonzero(s["src"] == src)[0]
            c = c[np.argsort(np.abs(np.log(s["colf"][c] / f)))[:3]]
            u = np.log(s["colf"][c])
            for i in range(3):
                o = [q for q in range(3) if q != i]
                out[:, j] += s["x"][:, c[i]] * np.prod([(np.log(f) - u[q]) / (u[i] - u[q]) for q in o])
        return out
    if kind in ("single", "forward") and case["model"] == "csem" and mesh.n_edges <= 15000:
        x = _exact_solve(s)
        return (x[:, 0].real.cpu().numpy(), x[:, 0].imag.cpu().numpy()) if kind == "single" else x
    return None
