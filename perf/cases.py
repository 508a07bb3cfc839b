"""The work a user's program has this framework do, as cases that can be timed and checked.

Kinds of case (``case["kind"]``):

* ``assemble``  A = K - k0^2 M on the device for a mesh whose pattern is known: one frequency of a
                solver loop (``GpuCSCMapping.to_device``). Small meshes (a filter model of 5k-13k
                tets, the serving stream's lower end), ordinary ones and the benchmark's box;
                isotropic, diagonal (PML) and full material tensors, with and without excluded
                conductor tets, in the three precisions.
* ``dropin``    the whole drop-in call of a driver that keeps everything on the host: materials and
                coordinates go in as numpy arrays, a ``scipy.sparse.csc_matrix`` comes out.
* ``setup``     a new mesh: its pattern and gather plan, its port term and its solve-DoF submatrix.
* ``driven``    one frequency of a driven two-port: A with the port term, the port's forcing vector
                and both reduced to the solve DoFs, on the device.
* ``sweep``     A(f) for a batch of frequencies from resident K and M, with the port term.
* ``heat``      the Lagrange-2 conduction and capacity matrices of a field, each to CSC values.
* ``fields``    the solution at points of known tets and the overlap integrals of a port face.
"""
import copy
import functools
import math

import numpy as np
import torch

from emerge_b200 import heat as H
from emerge_b200.assembly import GpuCSCMapping, tet_mass_stiffness_matrices
from emerge_b200.mesh import Nedelec2Field, TetMesh, plane_tris, structured_box
from emerge_b200.postprocess import FieldOnDevice, PortOverlap
from emerge_b200.robin import RobinTerm
from emerge_b200.serving import box_grid
from emerge_b200.solve_dofs import SolveSubmatrix
from emerge_b200.sweep import FrequencySweep

C0 = 299792458.0
WR90 = (22.86e-3, 10.16e-3, 50e-3)  # the waveguide box of the benchmark's configurations
HEAT_BOX = (0.1, 0.05, 0.067)


# ------------------------------------------------------------------ the cases
def listed():
    def c(name, kind, grid, **more):
        return dict(name=name, kind=kind, nx=grid[0], ny=grid[1], nz=grid[2], **more)

    return [
        # the smallest models of the serving stream (5k tets): launches and latency count
        c("assemble_5k_mixed", "assemble", (11, 5, 15), material="iso", precision="mixed", conductors=False),
        # the air-filled WR-90 box, one frequency of a small filter's loop
        c("assemble_13k_fp64", "assemble", (12, 6, 30), material="air", precision="fp64", conductors=False),
        # an anisotropic substrate (full tensors) around a metal post whose tets are left out; ragged sizes
        c("assemble_62k_full_fp64", "assemble", (23, 11, 41), material="full", precision="fp64", conductors=True),
        # a dielectric-loaded model at the upper end of the serving stream
        c("assemble_415k_mixed", "assemble", (48, 24, 60), material="iso", precision="mixed", conductors=False),
        # a box with a PML shell (diagonal complex tensors), the benchmark's million-tet size
        c("assemble_1008k_pml_fp64", "assemble", (84, 50, 40), material="pml", precision="fp64", conductors=False),
        # the benchmark's headline box
        c("assemble_2010k_fp64", "assemble", (100, 50, 67), material="iso", precision="fp64", conductors=False),
        # EMerge's own call, host arrays in and a scipy matrix out
        c("dropin_13k_fp64", "dropin", (12, 6, 30), material="iso", precision="fp64", conductors=False),
        # a new (refined) mesh: pattern, plan, port positions, solve-DoF slice
        c("setup_104k", "setup", (24, 12, 60), conductors=False),
        # one frequency of a driven two-port on the device
        c("driven_104k_fp64", "driven", (24, 12, 60), material="iso", precision="fp64", conductors=False),
        # twelve frequencies of a sweep in one call, as the benchmark's sweep forms them
        c("sweep_104k_12f", "sweep", (24, 12, 60), material="iso", precision="fp64", conductors=False, nf=12),
        # a conduction model: both matrices of a field
        c("heat_102k_fp64", "heat", (37, 18, 25), precision="fp64"),
        # a field plot of 200k points and the port integrals of its S-parameters
        c("fields_200k_points", "fields", (24, 12, 60), points=200_000),
    ]


def draw(rng):
    kind = rng.choice(["assemble"] * 5 + ["dropin", "setup", "driven", "sweep", "heat", "fields"])
    most = {"assemble": 5.9, "heat": 5.3}.get(kind, 5.1)
    n = 10 ** rng.uniform(3.7, most)
    nx, ny, nz = box_grid(int(n))
    nx, ny, nz = (max(2, v + rng.randint(-1, 2)) for v in (nx, ny, nz))
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind in ("assemble", "dropin", "driven", "sweep"):
        case["material"] = rng.choice(["iso", "iso", "air", "pml", "full"])
        case["precision"] = rng.choice(["fp64", "fp64", "mixed", "mixed", "exact"])
    if kind == "heat":
        case["precision"] = rng.choice(["fp64", "exact"])
    if kind in ("assemble", "dropin", "setup", "driven", "sweep"):
        # a port face has to keep its tets: the post of left-out tets ends below it
        case["conductors"] = rng.random() < 0.3
    if kind == "sweep":
        case["nf"] = rng.randint(1, 12)
    if kind == "fields":
        case["points"] = int(10 ** rng.uniform(3, 6))
    return case


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=2)
def _topology(nx, ny, nz, size):
    return TetMesh(*structured_box(nx, ny, nz, size=size, jitter=0.0))


def _mesh(case, rng, size, jitter=0.12):
    """The box's mesh with its interior vertices moved by up to 12% of a cell."""
    g = (case["nx"], case["ny"], case["nz"])
    m = copy.copy(_topology(*g, size))
    i = np.arange(m.n_nodes)
    at = (i % (g[0] + 1), (i // (g[0] + 1)) % (g[1] + 1), i // ((g[0] + 1) * (g[1] + 1)))
    nodes = m.nodes.copy()
    for d in range(3):
        move = rng.uniform(-jitter, jitter, m.n_nodes) * (size[d] / g[d])
        nodes[d] += np.where((at[d] > 0) & (at[d] < g[d]), move, 0.0)
    m.nodes = nodes
    return m


def _cells(case):
    """Grid cell (i, j, k) of every tet, six tets per cell, x fastest."""
    h = np.repeat(np.arange(case["nx"] * case["ny"] * case["nz"]), 6)
    return h % case["nx"], (h // case["nx"]) % case["ny"], h // (case["nx"] * case["ny"])


def _conductors(case):
    """The tets of a post through the middle of the box, clear of its end faces."""
    if not case.get("conductors"):
        return np.zeros(0, np.int64)
    i, j, k = _cells(case)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    inside = (abs(2 * i + 1 - nx) <= max(1, nx // 6)) & (j < max(1, ny // 2)) & (abs(2 * k + 1 - nz) <= max(1, nz // 6))
    return np.flatnonzero(inside).astype(np.int64)


def _materials(case, mesh, rng):
    """er, ur as EMerge passes them: c16[3, 3, n_tets]."""
    nT = mesh.n_tets
    er, ur = np.zeros((3, 3, nT), np.complex128), np.zeros((3, 3, nT), np.complex128)
    kind = case["material"]
    for d in range(3):
        er[d, d] = ur[d, d] = 1.0
    if kind in ("iso", "full"):
        i, j, k = _cells(case)  # one dielectric per block of 8 x 8 x 8 cells
        block = (i // 8) + 13 * ((j // 8) + 13 * (k // 8))
        n = int(block.max()) + 1
        eps = (rng.uniform(1.0, 10.0, n) * (1 - 1j * rng.uniform(1e-3, 1e-2, n)))[block]
        for d in range(3):
            er[d, d] = eps
    if kind == "full":  # reciprocal: symmetric complex tensors
        t = rng.uniform(-0.2, 0.2, (2, 3, 3, int(block.max()) + 1))
        t = (t + t.transpose(0, 2, 1, 3))[:, :, :, block]
        er *= np.eye(3)[:, :, None] + t[0] * (1 - 0.02j)
        er += t[0] * (1 - 0.02j)
        ur += t[1] * (1 - 0.01j)
    if kind == "pml":
        c = mesh.nodes[:, mesh.tets].mean(axis=1)
        k0 = 2 * np.pi * 10e9 / C0
        s = np.ones((3, nT), np.complex128)
        for d in range(3):
            depth = 0.1 * WR90[d]
            into = np.maximum(np.maximum(depth - c[d], c[d] - (WR90[d] - depth)), 0.0)
            s[d] -= 1j * (2.0 / depth) * rng.uniform(0.8, 1.2) * (into / depth) ** 2 / k0
        for d in range(3):
            er[d, d] = ur[d, d] = s[(d + 1) % 3] * s[(d + 2) % 3] / s[d]
    return er, ur


def _host(case, seed):
    """Everything a case's program holds on the host, from the seed alone."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "heat":
        mesh = _mesh(case, rng, HEAT_BOX)
        q = rng.normal(size=(3, 3, mesh.n_tets))
        cond = np.einsum("ijn,kjn->ikn", q, q) + 0.5 * np.eye(3)[:, :, None]
        return dict(mesh=mesh, field=H.Legrange2(mesh), cond=cond, rho=rng.uniform(1e6, 4e6, mesh.n_tets))
    mesh = _mesh(case, rng, WR90)
    h = dict(mesh=mesh, field=Nedelec2Field(mesh), freq=float(rng.uniform(8e9, 12e9)))
    if case["kind"] != "fields":
        h["conductors"] = _conductors(case)
    if "material" in case:
        h["er"], h["ur"] = _materials(case, mesh, rng)
    if case["kind"] in ("setup", "driven", "sweep", "fields"):
        h["ports"] = np.concatenate([plane_tris(mesh, 2, 0.0), plane_tris(mesh, 2, WR90[2])])
    N = h["field"].n_field
    if case["kind"] in ("setup", "driven"):
        walls = np.concatenate([plane_tris(mesh, d, v) for d in (0, 1) for v in (0.0, WR90[d])])
        edges = np.unique(mesh.tri_to_edge[:, walls])  # PEC walls: their DoFs are not solved for
        pec = np.concatenate([edges, edges + mesh.n_edges, walls + 2 * mesh.n_edges, walls + 2 * mesh.n_edges + mesh.n_tris])
        h["solve"] = np.setdiff1d(np.arange(N), pec)
    if case["kind"] in ("driven", "fields"):
        n = h["ports"].size
        te10 = np.sin(np.pi * mesh.nodes[0][mesh.tris[:, h["ports"]]].mean(axis=0) / WR90[0])
        U = 0.05 * (rng.normal(size=(3, 6, n)) + 1j * rng.normal(size=(3, 6, n)))
        U[1] += te10
        h["U"] = U
    if case["kind"] == "sweep":
        f = np.linspace(8e9, 12e9, case["nf"])
        h["coef"] = FrequencySweep.coefficients(f)
        h["gamma"] = 1j * np.sqrt((2 * np.pi * f / C0) ** 2 - (np.pi / WR90[0]) ** 2)
    if case["kind"] == "fields":
        h["x"] = rng.normal(size=N) + 1j * rng.normal(size=N)
        tet = rng.integers(0, mesh.n_tets, case["points"])
        bary = rng.exponential(size=(4, case["points"]))
        bary /= bary.sum(axis=0)
        h["tet"] = tet
        h["points"] = np.einsum("dvn,vn->dn", mesh.nodes[:, mesh.tets[:, tet]], bary)
    h["k0"] = 2 * np.pi * h["freq"] / C0
    h["port_gamma"] = 1j * math.sqrt(h["k0"] ** 2 - (np.pi / WR90[0]) ** 2)
    return h


def prepare(case, seed):
    h = _host(case, seed)
    kind, dev = case["kind"], torch.device("cuda", torch.cuda.current_device())
    s = dict(kind=kind, precision=case.get("precision"))
    if kind == "heat":
        s.update(field=h["field"], cond=h["cond"], rho=h["rho"])
    elif kind == "fields":
        s.update(fod=FieldOnDevice(h["field"]), points=h["points"], tet=h["tet"])
        s.update(x=torch.from_numpy(h["x"]).to(dev), U=torch.from_numpy(h["U"]).to(dev))
        s["overlap"] = PortOverlap(s["fod"], h["ports"])
    elif kind == "setup":
        s.update(field=h["field"], conductors=h["conductors"], ports=h["ports"], solve=h["solve"])
    else:
        E, B, cmap = tet_mass_stiffness_matrices(h["field"], h["er"], h["ur"], h["conductors"], precision=case["precision"])
        s.update(E=E, B=B, cmap=cmap, k0=h["k0"])
        if kind == "dropin":
            s.update(field=h["field"], er=h["er"], ur=h["ur"], conductors=h["conductors"])
        if kind in ("driven", "sweep"):
            s["port"] = RobinTerm(h["field"], h["ports"], cmap)
        if kind == "driven":
            s.update(gamma=h["port_gamma"], U=torch.from_numpy(h["U"]).to(dev), sub=SolveSubmatrix(cmap, h["solve"]))
        if kind == "sweep":
            s["sweep"] = FrequencySweep(E, B, cmap, robin=[s.pop("port")])
            s.update(coef=h["coef"], gamma=h["gamma"])
            s["out"] = torch.empty((case["nf"], cmap.nnz), dtype=torch.complex128, device=dev)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "assemble":
        return s["cmap"].to_device(s["E"] - s["B"] * s["k0"] ** 2)
    if kind == "dropin":
        E, B, cmap = tet_mass_stiffness_matrices(s["field"], s["er"], s["ur"], s["conductors"], s["cmap"],
                                                 precision=s["precision"])
        A = cmap.to_csc(E - B * s["k0"] ** 2)
        return [A.data, A.indices, A.indptr]
    if kind == "setup":
        cmap = GpuCSCMapping.from_field(s["field"], s["conductors"])
        port = RobinTerm(s["field"], s["ports"], cmap)
        sub = SolveSubmatrix(cmap, s["solve"])
        # the port term on the pattern: a program keeps it for its frequencies
        return [cmap.d_indptr, cmap.d_indices, port.to_device(1.0), sub.d_indptr[: sub.M + 1], sub.d_indices]
    if kind == "driven":
        A = s["cmap"].to_device(s["E"] - s["B"] * s["k0"] ** 2 + s["port"] * s["gamma"])
        b = s["port"].force(s["U"])
        return [A, b, s["sub"].values(A), s["sub"].rhs(b)]
    if kind == "sweep":
        return s["sweep"].form(s["coef"], out=s["out"], robin_gamma=s["gamma"])
    if kind == "heat":
        K, cmap = H.tet_stiffness_matrix(s["field"], s["cond"], precision=s["precision"])
        A = cmap.to_device(K)
        M, cmap = H.tet_mass_matrix(s["field"], s["rho"], precision=s["precision"])
        return [A, cmap.to_device(M), cmap.d_indptr, cmap.d_indices[: cmap.nnz]]
    E = s["fod"].interpolate(s["x"], s["points"], s["tet"])
    total, per = s["overlap"](s["x"], s["U"], 1.0)
    return [E, per, total.real, total.imag]


# ------------------------------------------------------------------ what a pass cannot do without
def _counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    V, T = (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz
    F = (4 * T + 4 * (nx * ny + ny * nz + nx * nz)) // 2
    return V, V + F - T - 1, F, T, 2 * nx * ny * 2  # nodes, edges, faces, tets, port triangles


def work(case):
    V, E, F, T, P = _counts(case)
    left = 1 - _conductors(case).size / T
    N, nnz = 2 * E + 2 * F, int(left * 4 * (E + 13 * F + 42 * T))
    tensor = {"air": 16, "iso": 16, "pml": 96, "full": 288}.get(case.get("material"), 0)
    mesh = 24 * V + 16 * T
    kind = case["kind"]
    if kind == "assemble":
        # per tet 210 entries of K and M from their two tensors, about 6 multiply-adds each
        return {"bytes": mesh + tensor * T * left + 16 * nnz, "flops": 2 * 2 * 210 * 6 * T * left}
    if kind == "dropin":
        return {"bytes": mesh + 288 * T + 20 * nnz + 4 * N, "flops": 2 * 2 * 210 * 6 * T * left}
    if kind == "setup":  # the topology in; both patterns and the port term on the pattern out
        return {"bytes": 40 * T + 4 * N + 4 * nnz + 16 * nnz + 4 * nnz + 4 * N, "flops": 64 * 6 * 4 * P}
    if kind == "driven":
        return {"bytes": mesh + tensor * T * left + 16 * nnz + 4 * nnz + 16 * nnz + 16 * N * 2,
                "flops": 2 * 2 * 210 * 6 * T * left}
    if kind == "sweep":
        return {"bytes": 32 * nnz + 16 * nnz * case["nf"], "flops": 8 * nnz * case["nf"]}
    if kind == "heat":
        n, pairs = V + E, V + 2 * E + 2 * E + 6 * F + 12 * T + E + 6 * F + 6 * T
        return {"bytes": 2 * mesh + 80 * T + 40 * T + 8 * pairs * 2 + 4 * pairs + 4 * n, "flops": 2 * 100 * 12 * T}
    n = case["points"]
    return {"bytes": n * (24 + 4 + 16 + 40 + 96 + 48) + 16 * N, "flops": n * 400}


# ------------------------------------------------------------------ the same in 64 bits, from the definitions
_EDGES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))  # vertex pairs, by rank of the global vertex number
_FACES = ((0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3))


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _basis(L, edges, faces):
    """c[point, function, vertex]: each function as sum_m c_m grad(lambda_m) at barycentrics L[point]."""
    n, nv = L.shape
    out = []
    for i, j in edges:
        c = np.zeros((n, nv))
        c[:, j], c[:, i] = L[:, i], -L[:, j]
        out.append(c)
    out += [(L[:, i] - L[:, j])[:, None] * c for (i, j), c in zip(edges, list(out))]
    for f, g in ((0, 1), (1, 0)):
        for t in faces:
            a, b, k = t[f], t[g], t[2]
            c = np.zeros((n, nv))
            c[:, k], c[:, b] = L[:, a] * L[:, b], -L[:, a] * L[:, k]
            out.append(c)
    return np.stack(out, axis=1)


def _curls(L):
    """c[point, function, pair]: each curl as sum_P c_P grad(lambda_i) x grad(lambda_j), P = (i, j)."""
    n = L.shape[0]
    where = {p: q for q, p in enumerate(_EDGES)}

    def add(c, i, j, v):
        if i != j:
            c[:, where[(min(i, j), max(i, j))]] += v if i < j else -v

    def product(c, a, b, k, v):  # curl of v * lambda_a lambda_b grad(lambda_k)
        add(c, a, k, v * L[:, b])
        add(c, b, k, v * L[:, a])

    out = []
    for i, j in _EDGES:
        c = np.zeros((n, 6))
        add(c, i, j, np.full(n, 2.0))
        out.append(c)
    for i, j in _EDGES:  # (Li - Lj)(Li grad Lj - Lj grad Li)
        c = np.zeros((n, 6))
        for a, b, k, v in ((i, i, j, 1.0), (i, j, i, -1.0), (j, i, j, -1.0), (j, j, i, 1.0)):
            product(c, a, b, k, v)
        out.append(c)
    for f, g in ((0, 1), (1, 0)):
        for t in _FACES:
            c = np.zeros((n, 6))
            product(c, t[f], t[g], t[2], 1.0)
            product(c, t[f], t[2], t[g], -1.0)
            out.append(c)
    return np.stack(out, axis=1)


def _cube_rule(dim):
    """Gauss-Legendre points of a simplex through the collapsed cube (degree 5 exact), weights summing to 1."""
    x, w = np.polynomial.legendre.leggauss(4)
    x, w = (x + 1) / 2, w / 2
    pts, wts = [], []
    for idx in np.ndindex(*(4,) * dim):
        left, lam, wt = 1.0, [], 1.0
        for d, q in enumerate(idx):
            lam.append(left * x[q])
            wt *= w[q] * (1 - x[q]) ** (dim - 1 - d)
            left *= 1 - x[q]
        pts.append([left] + lam)
        wts.append(wt * math.factorial(dim))
    return np.array(pts), np.array(wts)


def _gradients(nodes, tets):
    """(gradients [n, 4, 3], volume [n]) of the barycentrics, from edge vectors; tets [4, n]."""
    p = nodes[:, tets].permute(2, 1, 0)  # n, vertex, xyz
    e = p[:, 1:] - p[:, :1]
    c = torch.stack([torch.linalg.cross(e[:, 1], e[:, 2]), torch.linalg.cross(e[:, 2], e[:, 0]),
                     torch.linalg.cross(e[:, 0], e[:, 1])], dim=1)
    det = (e[:, 0] * c[:, 0]).sum(dim=1)
    g = c / det[:, None, None]
    return torch.cat([-g.sum(dim=1, keepdim=True), g], dim=1), det.abs() / 6


def _ranked(mesh, dev):
    """(tets with ascending vertex numbers [4, n], DoF of each canonical function [n, 20])."""
    tets, order = torch.sort(torch.from_numpy(mesh.tets).to(dev), dim=0)
    local = order.T  # n, rank -> the tet's own vertex
    t2e, t2t = torch.from_numpy(mesh.tet_to_edge).to(dev).T, torch.from_numpy(mesh.tet_to_tri).to(dev).T
    pair = torch.full((4, 4), -1, device=dev)
    for q, (i, j) in enumerate(((0, 1), (0, 2), (0, 3), (1, 2), (3, 1), (2, 3))):  # the mesh's edge slots
        pair[i, j] = pair[j, i] = q
    miss = torch.tensor([3, 1, 2, 0], device=dev)  # the face slot that lacks local vertex 0, 1, 2, 3
    e = torch.stack([t2e.gather(1, pair[local[:, i], local[:, j]][:, None])[:, 0] for i, j in _EDGES], dim=1)
    f = torch.stack([t2t.gather(1, miss[local[:, ({0, 1, 2, 3} - set(t)).pop()]][:, None])[:, 0] for t in _FACES], dim=1)
    E, F = mesh.n_edges, mesh.n_tris
    return tets, torch.cat([e, e + E, f + 2 * E, f + 2 * E + F], dim=1)


def _tables(dev):
    L, w = _cube_rule(3)
    c, k = _basis(L, _EDGES, _FACES), _curls(L)
    mass = np.einsum("q,qam,qbn->mnab", w, c, c).reshape(16, 400)
    stiff = np.einsum("q,qam,qbn->mnab", w, k, k).reshape(36, 400)
    return tuple(torch.from_numpy(x).to(dev) for x in (mass, stiff))


def _blocks(h, keep, tets, a, b):
    """a * stiffness + b * mass of the kept tets: complex [n, 400]."""
    dev = tets.device
    nodes = torch.from_numpy(h["mesh"].nodes).to(dev)
    mass, stiff = _tables(dev)
    pa = torch.tensor(_EDGES, device=dev)
    er, ur = (torch.from_numpy(h[k]).to(dev).permute(2, 0, 1)[keep] for k in ("er", "ur"))
    out = torch.empty((keep.numel(), 400), dtype=torch.complex128, device=dev)
    for lo in range(0, keep.numel(), 1 << 16):
        at = slice(lo, lo + (1 << 16))
        g, V = _gradients(nodes, tets[:, keep[at]])
        X = torch.linalg.cross(g[:, pa[:, 0]], g[:, pa[:, 1]]).to(torch.complex128)
        g = g.to(torch.complex128)
        G = torch.einsum("nxy,nmy,npx->nmp", er[at], g, g) * V[:, None, None]
        K = torch.einsum("nxy,nmy,npx->nmp", torch.linalg.inv(ur[at]), X, X) * V[:, None, None]
        out[at] = b * torch.complex(G.real.reshape(-1, 16) @ mass, G.imag.reshape(-1, 16) @ mass)
        out[at] += a * torch.complex(K.real.reshape(-1, 36) @ stiff, K.imag.reshape(-1, 36) @ stiff)
    return out


def _summed(keys, values):
    """(distinct keys ascending, summed values) of slots."""
    keys, order = torch.sort(keys)
    first = torch.ones_like(keys, dtype=torch.bool)
    first[1:] = keys[1:] != keys[:-1]
    to = torch.cumsum(first, 0) - 1
    out = torch.zeros(int(to[-1]) + 1, dtype=values.dtype, device=values.device)
    return keys[first], out.index_add_(0, to, values[order])


def _pattern_and(h, a, b):
    """(keys col * N + row, values) of a K + b M in CSC order."""
    dev, N = _device(), h["field"].n_field
    tets, dofs = _ranked(h["mesh"], dev)
    keep = np.delete(np.arange(h["mesh"].n_tets), h["conductors"])
    keep = torch.from_numpy(keep).to(dev)
    d = dofs[keep]
    keys = (d[:, None, :] * N + d[:, :, None]).reshape(-1)
    if a is None:
        return torch.unique(keys), None
    return _summed(keys, _blocks(h, keep, tets, a, b).reshape(-1))


def _port_parts(h):
    """(DoFs [n, 8], tangential basis table [6 points, 8, 3], gradients [n, 3, 3], area [n], points' weights)."""
    dev, m = _device(), h["mesh"]
    ids = torch.from_numpy(h["ports"]).to(dev)
    v = torch.from_numpy(m.nodes).to(dev)[:, torch.from_numpy(m.tris).to(dev)[:, ids]].permute(2, 1, 0)  # n, vertex, xyz
    e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    n2 = (nrm * nrm).sum(dim=1, keepdim=True)
    g1, g2 = torch.linalg.cross(e2, nrm) / n2, torch.linalg.cross(nrm, e1) / n2
    e = torch.from_numpy(m.tri_to_edge).to(dev)[:, ids].T
    E, F = m.n_edges, m.n_tris
    dofs = torch.cat([e, e + E, (ids + 2 * E)[:, None], (ids + 2 * E + F)[:, None]], dim=1)
    return dofs, torch.stack([-g1 - g2, g1, g2], dim=1), n2[:, 0].sqrt() / 2


_TRI_W = np.array([0.109951743655322] * 3 + [0.223381589678011] * 3)
_TRI_L = np.array([[0.81684757298045896, 0.09157621350977101, 0.09157621350977004],
                   [0.09157621350977101, 0.81684757298045896, 0.09157621350977008],
                   [0.09157621350977101, 0.09157621350977101, 0.81684757298045807],
                   [0.10810301816807, 0.445948490915965, 0.445948490915965],
                   [0.445948490915965, 0.10810301816807, 0.445948490915965],
                   [0.445948490915965, 0.445948490915965, 0.10810301816807]])  # the surface rule of degree 4
_TRI_EDGES, _TRI_FACE = ((0, 1), (1, 2), (0, 2)), ((0, 1, 2),)


def _port_on(h, keys):
    """The port term for gamma = 1 on the pattern's keys."""
    dofs, g, area = _port_parts(h)
    c = _basis(_TRI_L, _TRI_EDGES, _TRI_FACE)
    t = torch.from_numpy(np.einsum("q,qam,qbn->mnab", _TRI_W, c, c).reshape(9, 64)).to(g.device)
    B = torch.einsum("nmx,npx->nmp", g, g).reshape(-1, 9) @ t * area[:, None]
    N = h["field"].n_field
    k, v = _summed((dofs[:, None, :] * N + dofs[:, :, None]).reshape(-1), B.reshape(-1))
    out = torch.zeros(keys.numel(), dtype=torch.complex128, device=keys.device)
    out[torch.searchsorted(keys, k)] = v.to(torch.complex128)
    return out


def _force(h):
    dofs, g, area = _port_parts(h)
    c = torch.from_numpy(_basis(_TRI_L, _TRI_EDGES, _TRI_FACE)).to(g.device)
    U = torch.from_numpy(h["U"]).to(g.device)  # xyz, point, n
    w = torch.from_numpy(_TRI_W).to(g.device)
    gU = torch.einsum("nmx,xqn->nqm", g.to(torch.complex128), U)
    b = -area[:, None] * torch.einsum("q,qam,nqm->na", w.to(torch.complex128), c.to(torch.complex128), gU)
    out = torch.zeros(h["field"].n_field, dtype=torch.complex128, device=g.device)
    return out.index_add_(0, dofs.reshape(-1), b.reshape(-1))


def _solution_at(h, points, tet):
    """The solution at points [3, n] inside tets [n]: complex [3, n]."""
    dev = points.device
    tets, dofs = _ranked(h["mesh"], dev)
    nodes = torch.from_numpy(h["mesh"].nodes).to(dev)
    x = torch.from_numpy(h["x"]).to(dev)
    out = torch.empty((3, tet.numel()), dtype=torch.complex128, device=dev)
    for lo in range(0, tet.numel(), 1 << 18):
        at = slice(lo, lo + (1 << 18))
        own = tets[:, tet[at]]
        g, _ = _gradients(nodes, own)
        L = (g * (points[:, at].T - nodes[:, own[0]].T)[:, None]).sum(dim=2)
        L[:, 0] += 1
        y = x[dofs[tet[at]]]
        field = 0
        for n, (i, j) in enumerate(_EDGES):
            w = L[:, i, None] * g[:, j] - L[:, j, None] * g[:, i]
            field = field + w * (y[:, n] + (L[:, i] - L[:, j]) * y[:, 6 + n])[:, None]
        for n, (i, j, k) in enumerate(_FACES):
            field = field + (L[:, i] * y[:, 12 + n])[:, None] * (L[:, j, None] * g[:, k] - L[:, k, None] * g[:, j])
            field = field + (L[:, j] * y[:, 16 + n])[:, None] * (L[:, i, None] * g[:, k] - L[:, k, None] * g[:, i])
        out[:, at] = field.T
    return out


_HEAT_W = np.array([-0.078933] + [0.04573333] * 4 + [0.14933333] * 6)  # the 8-digit rule that defines the heat matrices
_A, _B, _C, _D = 0.78571429, 0.07142857, 0.39940358, 0.10059642
_HEAT_L = np.array([[0.25] * 4, [_A, _B, _B, _B], [_B, _B, _B, _A], [_B, _B, _A, _B], [_B, _A, _B, _B], [_C, _D, _C, _D],
                    [_C, _D, _D, _C], [_C, _C, _D, _D], [_D, _C, _C, _D], [_D, _C, _D, _C], [_D, _D, _C, _C]])


def _exact_heat(h):
    dev, f = _device(), h["field"]
    t = torch.from_numpy(h["mesh"].tets).to(dev)
    g, V = _gradients(torch.from_numpy(h["mesh"].nodes).to(dev), t)
    L = _HEAT_L
    n, dn = np.zeros((11, 10)), np.zeros((11, 10, 4))
    for i in range(4):
        n[:, i] = L[:, i] * (2 * L[:, i] - 1)
        dn[:, i, i] = 4 * L[:, i] - 1
    for e, (i, j) in enumerate(_EDGES):
        n[:, 4 + e] = 4 * L[:, i] * L[:, j]
        dn[:, 4 + e, i], dn[:, 4 + e, j] = 4 * L[:, j], 4 * L[:, i]
    mass = torch.from_numpy(np.einsum("q,qa,qb->ab", _HEAT_W, n, n).reshape(100)).to(dev)
    stiff = torch.from_numpy(np.einsum("q,qam,qbn->mnab", _HEAT_W, dn, dn).reshape(16, 100)).to(dev)
    cond = torch.from_numpy(h["cond"]).to(dev).permute(2, 0, 1)
    K = torch.einsum("nxy,nmy,npx->nmp", cond, g, g).reshape(-1, 16) @ stiff * V[:, None]
    M = (torch.from_numpy(h["rho"]).to(dev) * V)[:, None] * mass
    # the field's edge functions follow the mesh's edge slots (0,1), (0,2), (0,3), (1,2), (3,1), (2,3): the same pairs
    d = torch.from_numpy(f.tet_to_field).to(dev).T
    keys = (d[:, None, :] * f.n_field + d[:, :, None]).reshape(-1)
    return [_summed(keys, v.reshape(-1))[1] for v in (K, M)] + [None, None]


def exact(case, seed):
    kind = case["kind"]
    if 6 * case["nx"] * case["ny"] * case["nz"] > 450_000:
        return None  # the sort of its slots takes too long and too much memory
    h = _host(case, seed)
    if kind == "heat":
        return _exact_heat(h)
    if kind == "fields":
        dev = _device()
        E = _solution_at(h, torch.from_numpy(h["points"]).to(dev), torch.from_numpy(h["tet"]).to(dev))
        m, ids = h["mesh"], h["ports"]
        owner = np.full(m.n_tris, m.n_tets)
        np.minimum.at(owner, m.tet_to_tri.ravel(), np.tile(np.arange(m.n_tets), 4))
        v = torch.from_numpy(m.nodes[:, m.tris[:, ids]]).to(dev)  # xyz, vertex, n
        pts = torch.einsum("xvn,qv->xqn", v, torch.from_numpy(_TRI_L).to(dev))
        own = torch.from_numpy(owner[ids]).to(dev)
        at = _solution_at(h, pts.reshape(3, -1), own.repeat(6)).reshape(3, 6, -1)
        U = torch.from_numpy(h["U"]).to(dev)
        _, _, area = _port_parts(h)
        per = area * torch.einsum("q,xqn->n", torch.from_numpy(_TRI_W).to(dev).to(torch.complex128), (at - U) * U.conj())
        total = complex(per.sum())
        return [E, per, total.real, total.imag]
    if kind == "setup":
        keys, _ = _pattern_and(h, None, None)
        return [None, None, _port_on(h, keys), None, None]
    if kind == "sweep":
        keys, K = _pattern_and(h, 1.0, 0.0)
        _, M = _pattern_and(h, 0.0, 1.0)
        R = _port_on(h, keys)
        return torch.stack([K + c[2] * M + complex(g) * R for c, g in zip(h["coef"], h["gamma"])])
    keys, A = _pattern_and(h, 1.0, -h["k0"] ** 2)
    if kind == "assemble":
        return A
    if kind == "dropin":
        return [A.cpu().numpy(), None, None]
    A += h["port_gamma"] * _port_on(h, keys)
    b = _force(h)
    N = h["field"].n_field
    solve = torch.zeros(N, dtype=torch.bool, device=A.device)
    solve[torch.from_numpy(h["solve"]).to(A.device)] = True
    return [A, b, A[solve[keys // N] & solve[keys % N]], b[solve]]
