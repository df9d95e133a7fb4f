"""Timed workloads of the assembly library, through its public entry points.

A case is one call that a finite-element program makes many times on a mesh it keeps: an assembly
of the residual and the tangent, a residual alone, a matrix-free product, a Newton update, a new
sparsity pattern.  Its keys:

  call        "assemble" (residual + tangent), "residual", "action" (K v without K), "solve" (one
              Newton update: assembly + conjugate gradients), "pattern" (new Dirichlet conditions,
              new CSC pattern)
  physics     "poisson", "neohookean", "j2" (plasticity with state), "closure" (J2 with the learned
              closure at its plastic points)
  element     "quad4", "hex8", "tet4", "tet10", "hex27", or "mixed" (one block each of tet4, tet10
              and hex27, not connected to one another)
  nx, ny, nz  cells per direction (a cell holds one quad or hex, or six tets)
  distorted   corner nodes moved at random by up to 15% of the cell, as in a mesh of a part; else
              the box that the structured generator makes
  fixed       Dirichlet conditions on faces of the box (quad4 and hex8 meshes)
  precision   "fp64" or "fp32_element"
"""
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "finiteelementcontainers.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import fec_gb300 as fec  # noqa: E402
from fec_gb300 import closure as fec_closure  # noqa: E402

E, NU, SIGMA_Y, HARDENING = 200.0, 0.3, 0.25, 2.0   # J2: Young's modulus, Poisson ratio, yield stress, hardening
STRAIN = (0.005, 0.0055)                            # J2: the previous and the current load step's stretch
NNPE = {"quad4": 4, "hex8": 8, "tet4": 4, "tet10": 10, "hex27": 27}
NUM_Q = {"quad4": 4, "hex8": 8, "tet4": 1, "tet10": 4, "hex27": 27}
NAMES = {"quad4": "QUAD4", "hex8": "HEX8", "tet4": "TETRA4", "tet10": "TETRA10", "hex27": "HEX27"}


def _case(call, physics, element, cells, distorted=False, fixed=False, precision="fp64", **name):
    nx, ny, nz = (tuple(cells) + (1,))[:3]
    return dict(call=call, physics=physics, element=element, nx=nx, ny=ny, nz=nz, distorted=distorted, fixed=fixed,
                precision=precision, **name)


def listed():
    return [
        # the smallest problems: a 2D Poisson solve's assembly on a coarse grid, launch latency
        _case("assemble", "poisson", "quad4", (41, 29), fixed=True, name="poisson_quad4_small"),
        # the headline workload: Neo-Hookean on a structured box, all unknowns free
        _case("assemble", "neohookean", "hex8", (128, 128, 128), name="neohookean_hex8_box"),
        # the same physics on the mesh of a part (no two elements alike), clamped on one face
        _case("assemble", "neohookean", "hex8", (61, 53, 47), distorted=True, fixed=True,
              name="neohookean_hex8_part"),
        # the mixed-precision variant
        _case("assemble", "neohookean", "hex8", (96, 80, 88), precision="fp32_element", name="neohookean_hex8_fp32"),
        # residual alone: line searches, explicit steps, quasi-Newton
        _case("residual", "neohookean", "hex8", (67, 58, 71), distorted=True, fixed=True, name="residual_hex8_part"),
        # a load step of plasticity with state at every quadrature point
        _case("assemble", "j2", "hex8", (64, 56, 60), fixed=True, name="j2_hex8_box"),
        # the learned closure in place of the return map
        _case("assemble", "closure", "hex8", (44, 36, 40), fixed=True, precision="fp32_element",
              name="j2_closure_hex8"),
        # quadratic tets, the usual automatic mesh of a part
        _case("assemble", "neohookean", "tet10", (21, 19, 23), distorted=True, name="neohookean_tet10_part"),
        # several element types in one system
        _case("assemble", "neohookean", "mixed", (22, 24, 26), name="neohookean_mixed_box"),
        # matrix-free product of a Krylov method
        _case("action", "neohookean", "hex8", (72, 64, 68), name="action_hex8_box"),
        # one Newton update: assembly and the linear solve
        _case("solve", "poisson", "hex8", (36, 32, 34), fixed=True, name="solve_poisson_hex8"),
        # new Dirichlet conditions on a kept mesh: numbering and pattern again
        _case("pattern", "neohookean", "hex8", (48, 44, 52), fixed=True, name="pattern_hex8"),
    ]


def draw(rng):
    def cells(lo, hi):
        """Three sides whose cell count is spread over the logarithm of [lo, hi]."""
        side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1.0 / 3.0)
        return tuple(max(2, round(side * math.exp(rng.uniform(-0.35, 0.35)))) for _ in range(3))

    kind = rng.choice(("quad4", "poisson", "neohookean", "neohookean", "residual", "j2", "closure", "tets", "hex27",
                       "mixed", "action", "solve", "pattern"))
    bent = rng.random() < 0.5
    fixed = rng.random() < 0.5
    precision = "fp32_element" if rng.random() < 0.3 else "fp64"
    if kind == "quad4":
        return _case("assemble", "poisson", "quad4", tuple(round(math.exp(rng.uniform(2.0, 6.2))) for _ in range(2)),
                     distorted=bent, fixed=True)
    if kind == "poisson":
        return _case("assemble", "poisson", "hex8", cells(50, 300_000), distorted=bent, fixed=True)
    if kind == "neohookean":
        return _case("assemble", "neohookean", "hex8", cells(50, 500_000), distorted=bent, fixed=fixed,
                     precision=precision)
    if kind == "residual":
        return _case("residual", "neohookean", "hex8", cells(50, 500_000), distorted=bent, fixed=fixed,
                     precision=precision)
    if kind == "j2":
        return _case("assemble", "j2", "hex8", cells(50, 250_000), distorted=bent, fixed=True, precision=precision)
    if kind == "closure":
        return _case("assemble", "closure", "hex8", cells(50, 80_000), distorted=bent, fixed=True,
                     precision="fp32_element")
    if kind == "tets":
        return _case("assemble", "neohookean", rng.choice(("tet4", "tet10")), cells(20, 12_000), distorted=bent,
                     precision=precision)
    if kind == "hex27":
        return _case("assemble", "neohookean", "hex27", cells(20, 12_000), distorted=bent, precision=precision)
    if kind == "mixed":
        return _case("assemble", "neohookean", "mixed", cells(20, 12_000), distorted=bent, precision=precision)
    if kind == "action":
        return _case("action", "neohookean", "hex8", cells(50, 500_000), distorted=bent, fixed=fixed)
    if kind == "solve":
        return _case("solve", "poisson", "hex8", cells(50, 100_000), distorted=bent, fixed=True)
    return _case("pattern", "neohookean", "hex8", cells(50, 200_000), distorted=bent, fixed=True)


# -- meshes (numpy, 0-based; nodes with x fastest) -----------------------------------------------------------------

HEX = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1))
TETS = ((0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6))   # around the diagonal
EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))


def _line(n):
    t = np.arange(n + 1) / n
    return (1.0 - t) * 0.0 + t * 1.0


def _grid(counts):
    """Coordinates of the nodes of a unit box with counts[d] intervals."""
    ax = np.meshgrid(*[_line(n) for n in reversed(counts)], indexing="ij")
    return np.stack([x.ravel() for x in reversed(ax)], 1)


def _moves(cells, seed):
    """Random moves of the corner nodes, up to 15% of the cell, on the corner grid (nz+1, ny+1, nx+1, dim)."""
    r = np.random.default_rng(seed)
    return r.uniform(-0.15, 0.15, [n + 1 for n in reversed(cells)] + [len(cells)]) / np.array(cells, dtype=float)


def _refined(m):
    """A corner field on the grid with a node between any two neighbours."""
    for d in range(m.ndim - 1):
        m = np.moveaxis(m, d, 0)
        out = np.empty((2 * m.shape[0] - 1,) + m.shape[1:])
        out[::2] = m
        out[1::2] = 0.5 * (m[1:] + m[:-1])
        m = np.moveaxis(out, 0, d)
    return m


@functools.lru_cache(maxsize=8)
def _connectivity(element, cells):
    """(NE, NNPE) node numbers."""
    n = cells
    if element == "quad4":
        ey, ex = (v.ravel() for v in np.meshgrid(np.arange(n[1]), np.arange(n[0]), indexing="ij"))
        return np.stack([ex + i + (n[0] + 1) * (ey + j) for i, j in ((0, 0), (1, 0), (1, 1), (0, 1))], 1)
    if element == "hex8":   # elements with z fastest, as the structured generator numbers them
        ex, ey, ez = (v.ravel() for v in np.meshgrid(*[np.arange(k) for k in n], indexing="ij"))
        return np.stack([ex + i + (n[0] + 1) * (ey + j + (n[1] + 1) * (ez + k)) for i, j, k in HEX], 1)
    ez, ey, ex = (v.ravel() for v in np.meshgrid(*[np.arange(k) for k in reversed(n)], indexing="ij"))
    s = 1 if element == "tet4" else 2
    at = lambda i, j, k: s * ex + i + (s * n[0] + 1) * (s * ey + j + (s * n[1] + 1) * (s * ez + k))  # noqa: E731
    if element == "hex27":
        return np.stack([at(i, j, k) for k in range(3) for j in range(3) for i in range(3)], 1)
    tets = []
    for t in TETS:
        c = np.array([HEX[v] for v in t])
        if np.linalg.det(c[1:] - c[0]) < 0:
            c[[1, 2]] = c[[2, 1]]
        nodes = [at(*(s * v)) for v in c]
        if element == "tet10":
            nodes += [at(*(c[i] + c[j])) for i, j in EDGES]
        tets.append(np.stack(nodes, 1))
    return np.stack(tets, 1).reshape(-1, NNPE[element])


def _mesh(element, cells, seed):
    """(coordinates, connectivity); seed None: the undistorted box."""
    conn = _connectivity(element, cells)
    if element in ("quad4", "hex8", "tet4"):
        X = _grid(cells)
        if seed is not None:
            X = X + _moves(cells, seed).reshape(X.shape)
    else:
        X = _grid([2 * n for n in cells])
        if seed is not None:
            X = X + _refined(_moves(cells, seed)).reshape(X.shape)
            if element == "tet10":   # straight edges: mid nodes halfway between the corners
                for e, (i, j) in enumerate(EDGES):
                    X[conn[:, 4 + e]] = 0.5 * (X[conn[:, i]] + X[conn[:, j]])
    return X, conn


def _blocks(case, seed):
    """(coordinates, [(element, connectivity)]) of a case."""
    cells = (case["nx"], case["ny"]) if case["element"] == "quad4" else (case["nx"], case["ny"], case["nz"])
    kinds = ("tet4", "tet10", "hex27") if case["element"] == "mixed" else (case["element"],)
    Xs, blocks, at = [], [], 0
    for i, kind in enumerate(kinds):
        X, conn = _mesh(kind, cells, seed * 3 + i if case["distorted"] else None)
        Xs.append(X)
        blocks.append((kind, conn + at))
        at += len(X)
    return np.concatenate(Xs), blocks


def _faces(case):
    """Nodes of the box's faces (quad4 and hex8 meshes), 0-based."""
    if case["element"] not in ("quad4", "hex8"):
        return {}
    n = [case["nx"], case["ny"]] + ([case["nz"]] if case["element"] == "hex8" else [])
    ids = np.arange(np.prod([k + 1 for k in n])).reshape([k + 1 for k in reversed(n)])
    out = {}
    for d, (lo, hi) in enumerate((("left", "right"), ("bottom", "top"), ("back", "front"))[:len(n)]):
        out[lo] = np.take(ids, 0, axis=len(n) - 1 - d).ravel()
        out[hi] = np.take(ids, -1, axis=len(n) - 1 - d).ravel()
    return out


# -- inputs ---------------------------------------------------------------------------------------------------------

def _field(case, X, seed, step=1):
    """The nodal field (NN, NF): Uniform[-1, 1] for Poisson, a stretch with noise for Neo-Hookean (a twentieth of
    the cell, less where nodes are closer than that), load step `step` of a uniaxial stretch for J2."""
    r = np.random.default_rng(1000 * seed + step)
    if case["physics"] == "poisson":
        return r.uniform(-1.0, 1.0, (len(X), 1))
    if case["physics"] == "neohookean":
        noise = (0.05 if case["element"] == "hex8" else 0.02) / max(case["nx"], case["ny"], case["nz"])
        return X * np.array([0.05, -0.02, -0.02]) + noise * r.standard_normal(X.shape)
    e = STRAIN[step]
    return X * np.array([e, -NU * e, -NU * e]) + 1e-5 * r.standard_normal(X.shape)


def _fixed(case, step=1):
    """[(component, face, value(X))] of the Dirichlet conditions."""
    if not case["fixed"]:
        return []
    if case["physics"] == "poisson":
        return [(0, f, lambda X: 0.0) for f in _faces(case)]
    if case["physics"] == "neohookean":
        return [(i, "left", lambda X: 0.0) for i in range(3)]
    return [(0, "left", lambda X: 0.0), (1, "bottom", lambda X: 0.0), (2, "back", lambda X: 0.0),
            (0, "right", lambda X: STRAIN[step] * X[0])]


def _physics(case):
    if case["physics"] == "poisson":
        return fec.Poisson(1.0)
    if case["physics"] == "neohookean":
        return fec.NeoHookean.from_youngs(1.0, 0.3)
    if case["physics"] == "j2":
        return fec.J2Plasticity(E, NU, SIGMA_Y, HARDENING)
    return fec_closure.J2Closure(E, NU, SIGMA_Y, HARDENING, _trained())


@functools.lru_cache(maxsize=1)
def _trained():
    """A small closure, trained once in a process and kept, as a program keeps its weights."""
    X, Y, plastic = fec_closure.generate_samples([E, NU, SIGMA_Y, HARDENING], n_paths=6000, steps=10, seed=4)
    return fec_closure.train(X[plastic], Y[plastic], epochs=8, batch=2048, lr=5e-3, tol=1e-2)


def prepare(case, seed):
    X, blocks = _blocks(case, seed)
    mesh = fec.UnstructuredMesh(X, {k: (NAMES[k], conn + 1) for k, conn in blocks},
                                {k: v + 1 for k, v in _faces(case).items()})
    space = fec.FunctionSpace(mesh)
    scalar = case["physics"] == "poisson"
    u = fec.ScalarFunction(space, "u") if scalar else fec.VectorFunction(space, "u")
    asm = fec.SparseMatrixAssembler(u, precision=case["precision"],
                                    symbolic="device" if case["call"] == "pattern" else "host")

    def conditions(step):
        return [fec.DirichletBC(u.names[i], lambda x, t, v=value: v(x), nodeset_name=face)
                for i, face, value in _fixed(case, step)]

    old = case["physics"] in ("j2", "closure")
    p = fec.create_parameters(mesh, asm, _physics(case), dirichlet_bcs=conditions(0 if old else 1))
    free = torch.from_numpy(asm.dof.unknown_dofs - 1)

    def unknowns(step):
        return torch.from_numpy(_field(case, X, seed, step).ravel())[free].cuda()

    if old:   # the previous load step leaves its plastic strains behind
        fec.assemble_vector(asm, fec.residual, unknowns(0), p)
        p.swap_states()
        p.dirichlet_bcs = conditions(1)
        p.update_bc_values()
    state = {"case": case, "asm": asm, "p": p, "Uu": unknowns(1)}
    if case["call"] == "action":
        g = torch.Generator().manual_seed(seed)
        state["Vu"] = torch.randn(len(free), generator=g, dtype=torch.float64).cuda()
    elif case["call"] == "solve":
        state["solver"] = fec.IterativeLinearSolver(asm, rtol=1e-12)
    elif case["call"] == "pattern":
        # the next change of the conditions holds one component of one more face
        state["bcs"] = conditions(1) + [fec.DirichletBC(u.names[seed // 2 % 3], lambda x, t: 0.0,
                                                        nodeset_name=("bottom", "top")[seed % 2])]
    if case["call"] != "pattern":
        asm.pattern()
    return state


def run(state):
    case, asm, p, Uu = state["case"], state["asm"], state["p"], state["Uu"]
    if case["call"] == "assemble":
        R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
        out = {"residual": R, "nzval": K.nzval}
        if case["physics"] in ("j2", "closure"):
            out["state"] = p.state_new
        return out
    if case["call"] == "residual":
        fec.assemble_vector(asm, fec.residual, Uu, p)
        return {"residual": fec.residual(asm)}
    if case["call"] == "action":
        fec.assemble_matrix_free_action(asm, fec.stiffness_action, Uu, state["Vu"], p)
        return {"action": fec.hvp(asm)}
    if case["call"] == "solve":
        return {"unknowns": state["solver"].solve(Uu.clone(), p)}
    fec.update_dofs_bcs(asm, state["bcs"])
    colptr, rowval = asm.pattern_device()
    return {"colptr": colptr, "rowval": rowval}


# -- the work that a pass cannot do without ---------------------------------------------------------------------------

def _sizes(case):
    """[(element, elements, nodes, neighbouring (node, node) pairs)] per block of the undivided box."""
    n = [case["nx"], case["ny"], case["nz"]]
    kinds = ("tet4", "tet10", "hex27") if case["element"] == "mixed" else (case["element"],)
    out = []
    for kind in kinds:
        if kind == "quad4":
            out.append((kind, n[0] * n[1], (n[0] + 1) * (n[1] + 1), (3 * n[0] + 1) * (3 * n[1] + 1)))
            continue
        c = math.prod(n)
        if kind == "hex8":
            out.append((kind, c, math.prod(k + 1 for k in n), math.prod(3 * k + 1 for k in n)))
        elif kind == "hex27":   # 1D: corner nodes see 5 nodes (3 at the ends), mid nodes 3
            out.append((kind, c, math.prod(2 * k + 1 for k in n), math.prod(8 * k + 1 for k in n)))
        elif kind == "tet4":
            out.append((kind, 6 * c, math.prod(k + 1 for k in n), 15 * math.prod(k + 1 for k in n)))
        else:
            out.append((kind, 6 * c, math.prod(2 * k + 1 for k in n), 28 * math.prod(2 * k + 1 for k in n)))
    return out


def work(case):
    """Bytes: connectivity (4 B a node number), coordinates and fields read once, outputs written once.  Flops: of the
    element integrals (symmetric tangents), not of the index work."""
    nf = 1 if case["physics"] == "poisson" else 3
    dim = 2 if case["element"] == "quad4" else 3
    state = 2 * 7 * 8 if case["physics"] in ("j2", "closure") else 0   # bytes per quadrature point, read and written
    nbytes = flops = 0.0
    for kind, ne, nn, pairs in _sizes(case):
        a, q = NNPE[kind], NUM_Q[kind]
        nnz = nf * nf * pairs
        if case["call"] == "pattern":
            nbytes += 4 * a * ne + 8 * nf * nn + 8 * nf * nn + 8 * nnz
            continue
        point = 2 * a * dim * dim + 60 + 2 * a * nf * dim + (200 if nf == 3 else 20)   # map, gradient, material
        force = 2 * a * nf * dim
        tangent = (162 * a + 54 * a * (a + 1) / 2) if nf == 3 else dim * a * (a + 1)
        nbytes += 4 * a * ne + 8 * dim * nn + 8 * nf * nn + state * q * ne + 8 * nf * nn
        if case["call"] == "residual":
            flops += ne * q * (point + force)
        elif case["call"] == "action":
            nbytes += 8 * nf * nn
            flops += ne * q * (point + 2 * a * nf * dim + 100 + force)
        else:
            flops += ne * q * (point + force + tangent)
            nbytes += 8 * nnz
            if case["call"] == "solve":   # every iteration reads the matrix and its row numbers; about 3 a side
                its = 3 * max(case["nx"], case["ny"], case["nz"])
                nbytes += its * (12 * nnz + 8 * 8 * nn)
                flops += its * 2 * nnz
    return {"bytes": nbytes, "flops": flops}


# -- the same results in 64 bits, by plain torch ----------------------------------------------------------------------

def _points(kind):
    """(points, weights) of the rules that the calls use: 2 and 3 points a direction, 1 and 4 in a tet."""
    if kind == "tet4":
        return np.full((1, 3), 0.25), np.array([1 / 6])
    if kind == "tet10":
        lo = (5 - math.sqrt(5)) / 20
        return np.full((4, 3), lo) + np.vstack([np.zeros(3), (1 - 4 * lo) * np.eye(3)]), np.full(4, 1 / 24)
    g, w = np.polynomial.legendre.leggauss(3 if kind == "hex27" else 2)
    dim = 2 if kind == "quad4" else 3
    at = np.meshgrid(*[np.arange(len(g))] * dim, indexing="ij")
    at = [k.ravel() for k in reversed(at)]   # x fastest
    return np.stack([g[k] for k in at], 1), np.prod([w[k] for k in at], axis=0)


def _shapes(kind):
    """Shape functions N (NQ, A), gradients dN (NQ, A, dim), weights."""
    pts, w = _points(kind)
    if kind in ("tet4", "tet10"):
        lam = np.concatenate([1 - pts.sum(1, keepdims=True), pts], 1)
        dl = np.vstack([-np.ones(3), np.eye(3)])
        if kind == "tet4":
            return lam, np.broadcast_to(dl, (1, 4, 3)).copy(), w
        N = np.concatenate([lam * (2 * lam - 1)] + [4 * lam[:, [i]] * lam[:, [j]] for i, j in EDGES], 1)
        dN = [(4 * lam[:, v, None] - 1) * dl[v] for v in range(4)]
        dN += [4 * (lam[:, j, None] * dl[i] + lam[:, i, None] * dl[j]) for i, j in EDGES]
        return N, np.stack(dN, 1), w
    if kind == "hex27":
        nodes = [(i, j, k) for k in range(3) for j in range(3) for i in range(3)]
        f = lambda x: np.stack([x * (x - 1) / 2, 1 - x * x, x * (x + 1) / 2], -1)  # noqa: E731
        d = lambda x: np.stack([x - 0.5, -2 * x, x + 0.5], -1)  # noqa: E731
    else:
        nodes = HEX if kind == "hex8" else [h[:2] for h in HEX[:4]]
        f = lambda x: np.stack([(1 - x) / 2, (1 + x) / 2], -1)  # noqa: E731
        d = lambda x: np.stack([-0.5 + 0 * x, 0.5 + 0 * x], -1)  # noqa: E731
    dim = pts.shape[1]
    val, der = [f(pts[:, k]) for k in range(dim)], [d(pts[:, k]) for k in range(dim)]
    pick = lambda t: np.stack([np.prod([t[k][:, n[k]] for k in range(dim)], axis=0) for n in nodes], 1)  # noqa: E731
    grads = [pick([der[k] if k == j else val[k] for k in range(dim)]) for j in range(dim)]
    return pick(val), np.stack(grads, 2), w


def _inverse(F):
    """(determinant, inverse) of 2 x 2 or 3 x 3 matrices."""
    if F.shape[-1] == 2:
        (a, b), (c, d) = F[..., 0, :].unbind(-1), F[..., 1, :].unbind(-1)
        det = a * d - b * c
        return det, torch.stack([d, -b, -c, a], -1).reshape(F.shape) / det[..., None, None]
    a, b, c = F.unbind(-2)
    cof = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], -1)
    det = (a * cof[..., 0]).sum(-1)
    return det, cof / det[..., None, None]


def _neohookean(F, want):
    """P (.., 3, 3) and A (.., 3, 3, 3, 3) of psi = K/2 ((J-1)^2/2 - ln J) + G/2 (J^(-2/3) F:F - 3)."""
    K, G = 1.0 / (3 * (1 - 0.6)), 1.0 / 2.6
    J, H = _inverse(F)
    J, H = J[..., None, None], H.transpose(-1, -2)
    I1 = (F * F).sum((-1, -2), keepdim=True)
    c1, c2 = 0.5 * K * (J * J - J - 1), G * J.pow(-2.0 / 3.0)
    P = c1 * H + c2 * (F - I1 / 3 * H)
    if not want:
        return P, None
    o = lambda a, b: a[..., :, :, None, None] * b[..., None, None, :, :]  # noqa: E731
    s = lambda c: c[..., None, None]  # noqa: E731
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    A = s(0.5 * K * (2 * J - 1) * J + 2.0 / 9.0 * c2 * I1) * o(H, H)
    A += s(I1 / 3 * c2 - c1) * torch.einsum("...il,...kj->...ijkl", H, H)
    A += s(c2) * torch.einsum("ik,jl->ijkl", eye, eye) - s(2.0 / 3.0 * c2) * (o(F, H) + o(H, F))
    return P, A


def _j2(gu, state, want):
    """Stress, tangent and new state (.., 7) of the radial return; state: plastic strain xx yy zz yz xz xy, eqps."""
    mu, kappa = E / (2 * (1 + NU)), E / (3 * (1 - 2 * NU))
    eye = torch.eye(3, dtype=gu.dtype, device=gu.device)
    ix = torch.tensor([[0, 5, 4], [5, 1, 3], [4, 3, 2]], device=gu.device)
    eps = 0.5 * (gu + gu.transpose(-1, -2))
    etr = eps - state[..., :6][..., ix]
    tr = etr.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None]
    s = 2 * mu * (etr - tr / 3 * eye)
    norm = (s * s).sum((-1, -2), keepdim=True).sqrt()
    f = norm - math.sqrt(2 / 3) * (SIGMA_Y + HARDENING * state[..., 6, None, None])
    plastic = f > 0
    dg = torch.where(plastic, f / (2 * mu + 2 / 3 * HARDENING), 0.0)
    n = s / norm.clamp_min(1e-300)
    P = kappa * tr * eye + s - 2 * mu * dg * n
    ep = dg * n
    step = torch.stack([ep[..., 0, 0], ep[..., 1, 1], ep[..., 2, 2], ep[..., 1, 2], ep[..., 0, 2], ep[..., 0, 1],
                        math.sqrt(2 / 3) * dg[..., 0, 0]], -1)
    if not want:
        return P, None, state + step
    theta = 1 - 2 * mu * dg / norm.clamp_min(1e-300)
    bar = torch.where(plastic, 1 / (1 + HARDENING / (3 * mu)) - (1 - theta), 0.0)
    sym = 0.5 * (torch.einsum("ik,jl->ijkl", eye, eye) + torch.einsum("il,jk->ijkl", eye, eye))
    vol = torch.einsum("ij,kl->ijkl", eye, eye)
    w = lambda c: c[..., None, None]  # noqa: E731
    A = kappa * vol + 2 * mu * w(theta) * (sym - vol / 3) - 2 * mu * w(bar) * n[..., :, :, None, None] * n[..., None, None, :, :]
    return P, A, state + step


def _elements(case, kind, X, U, state, want):
    """Element residuals (E, A, NF), tangents (E, A, NF, A, NF) or None, new states or None, of gathered X and U."""
    N, dN, w = (torch.from_numpy(v).to(X) for v in _shapes(kind))
    det, inverse = _inverse(torch.einsum("eai,qaj->eqij", X, dN))
    grad = torch.einsum("qaj,eqji->eqai", dN, inverse)
    jxw = det * w
    gu = torch.einsum("eai,eqaj->eqij", U, grad)
    new = None
    if case["physics"] == "poisson":
        source = torch.sin(math.pi * torch.einsum("qa,eai->eqi", N, X)).prod(-1)
        R = torch.einsum("eq,eqaj,eqj->ea", jxw, grad, gu[:, :, 0]) - torch.einsum("eq,qa->ea", jxw * source, N)
        K = torch.einsum("eq,eqaj,eqbj->eab", jxw, grad, grad)[:, :, None, :, None] if want else None
        return R[..., None], K, new
    if case["physics"] == "neohookean":
        P, A = _neohookean(gu + torch.eye(3).to(X), want)
    else:
        P, A, new = _j2(gu, state, want)
    R = torch.einsum("eq,eqij,eqaj->eai", jxw, P, grad)
    if not want:
        return R, None, new
    ne, nq, na = grad.shape[:3]
    left = torch.einsum("eqaj,eqijkl->eqaikl", grad, A * jxw[..., None, None, None, None])
    # sum over (q, l) as one product of (a i k, q l) and (q l, b)
    left = left.permute(0, 2, 3, 4, 1, 5).reshape(ne, na * 9, nq * 3)
    K = torch.bmm(left, grad.transpose(2, 3).reshape(ne, nq * 3, na)).reshape(ne, na, 3, 3, na)
    return R, K.transpose(3, 4), new


def _pattern_of(blocks, free, nn, nf):
    """Positions in the CSC values: per block pair numbers (E, A, A) of (column node, row node), and per pair the place
    of its first entry, per column node the length of its columns."""
    keys = [(c[:, :, None] * nn + c[:, None, :]) for c in blocks]
    uniq, inv = torch.unique(torch.cat([k.reshape(-1) for k in keys]), return_inverse=True)
    col, row = uniq // nn, uniq % nn
    count = free.sum(1)
    rows = count[row]
    length = torch.zeros(nn, dtype=torch.int64, device=free.device).index_add_(0, col, rows)
    before = rows.cumsum(0) - rows
    entries = count * length
    base = entries.cumsum(0) - entries
    offset = before - (length.cumsum(0) - length)[col]
    split = inv.split([k.numel() for k in keys])
    return [s.reshape(k.shape) for s, k in zip(split, keys)], base[col] + offset, length[col], int(entries.sum())


def exact(case, seed):
    if case["physics"] == "closure" or case["call"] == "pattern":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X, blocks = _blocks(case, seed)
    nn, nf = len(X), 1 if case["physics"] == "poisson" else 3
    fields, faces = [], _faces(case)
    for step in (0, 1):
        U = _field(case, X, seed, step)
        for i, face, value in _fixed(case, step):
            U[faces[face], i] = [value(x) for x in X[faces[face]]]
        fields.append(torch.from_numpy(U).to(dev))
    free = np.ones((nn, nf), dtype=bool)
    for i, face, _ in _fixed(case):
        free[faces[face], i] = False
    free = torch.from_numpy(free).to(dev)
    X, conns = torch.from_numpy(X).to(dev), [torch.from_numpy(c).to(dev) for _, c in blocks]
    want = case["call"] != "residual"
    R = torch.zeros(nn, nf, dtype=torch.float64, device=dev)
    V = torch.zeros_like(R)
    if case["call"] == "action":
        g = torch.Generator().manual_seed(seed)
        V[free] = torch.randn(int(free.sum()), generator=g, dtype=torch.float64).to(dev)
    matrix = case["call"] in ("assemble", "solve")
    if matrix:
        pair, first, length, nnz = _pattern_of(conns, free, nn, nf)
        nzval = torch.zeros(nnz, dtype=torch.float64, device=dev)
        rank = free.cumsum(1) - 1
    states = []
    for b, (kind, conn) in enumerate(zip([k for k, _ in blocks], conns)):
        chunk = 32_000_000 // NNPE[kind] ** 2 // NUM_Q[kind] + 1
        for at in range(0, len(conn), chunk):
            c = conn[at:at + chunk]
            state = None
            if case["physics"] == "j2":
                state = torch.zeros(len(c), NUM_Q[kind], 7, dtype=torch.float64, device=dev)
                state = _elements(case, kind, X[c], fields[0][c], state, False)[2]
            Re, Ke, new = _elements(case, kind, X[c], fields[1][c], state, want)
            if new is not None:
                states.append(new.reshape(-1))
            if case["call"] == "action":
                Re = torch.einsum("eaibk,ebk->eai", Ke, V[c])
            R.index_add_(0, c.reshape(-1), Re.reshape(-1, nf))
            if matrix:
                p = pair[b][at:at + chunk]
                for k in range(nf):       # column component
                    for i in range(nf):   # row component
                        ok = free[c][:, :, None, k] & free[c][:, None, :, i]
                        place = first[p] + rank[c][:, :, None, k] * length[p] + rank[c][:, None, :, i]
                        nzval.index_add_(0, place[ok], Ke[:, :, i, :, k].transpose(1, 2)[ok])
    if case["call"] == "residual":
        return {"residual": R[free]}
    if case["call"] == "action":
        return {"action": R[free]}
    if case["call"] == "assemble":
        out = {"residual": R[free], "nzval": nzval}
        return out | ({"state": torch.cat(states)} if states else {})
    # the update of a linear problem: conjugate gradients on the matrix, far below the caller's tolerance
    counts = torch.zeros(nn, dtype=torch.int64, device=dev)
    column = torch.unique(conns[0][:, :, None] * nn + conns[0][:, None, :])
    column = column[free[column // nn, 0] & free[column % nn, 0]]
    counts.index_add_(0, column // nn, torch.ones_like(column))
    number = rank.new_zeros(nn)
    number[free[:, 0]] = torch.arange(int(free.sum()), device=dev)
    ptr = torch.cat([counts.new_zeros(1), counts[free[:, 0]].cumsum(0)])
    K = torch.sparse_csr_tensor(ptr, number[column % nn], nzval, (len(ptr) - 1,) * 2, check_invariants=False)
    b = R[free]
    x, r = torch.zeros_like(b), b.clone()
    d, rr = r.clone(), r.dot(r)
    for _ in range(4000):
        Kd = K @ d
        alpha = rr / d.dot(Kd)
        x += alpha * d
        r -= alpha * Kd
        new = r.dot(r)
        if float(new) <= 1e-30 * float(b.dot(b)):
            break
        d, rr = r + (new / rr) * d, new
    return {"unknowns": fields[1][free] - x}
