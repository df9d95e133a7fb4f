"""FP64 Neo-Hookean hex8 blocks of any shape on the tensor cores (the contraction in
reference coordinates) against the CPU oracle and the per-element kernels: tile edges
(12 elements a tile), flat and skewed elements, permuted local numberings, Lobatto
points, Dirichlet dofs, and the calls and workspaces that must agree bitwise."""
import os

import numpy as np
import pytest

from helpers import blocks_of, rel_err, residual_err

pytestmark = pytest.mark.gpu
TOL64 = 1e-12
# rotations of the reference cube as node orders (each keeps the orientation)
ORDERS = ([0, 1, 2, 3, 4, 5, 6, 7], [1, 2, 3, 0, 5, 6, 7, 4], [4, 0, 3, 7, 5, 1, 2, 6], [6, 5, 4, 7, 2, 1, 0, 3])


def _mesh(fec, cells, seed, stretch=(1.0, 1.0, 1.0), rotate=False):
    ax = [np.linspace(0.0, s, n + 1) for n, s in zip(cells, stretch)]
    z, y, x = np.meshgrid(*ax[::-1], indexing="ij")
    X = np.stack([x.ravel(), y.ravel(), z.ravel()], 1)
    rng = np.random.default_rng(seed)
    X = X + rng.uniform(-0.2, 0.2, X.shape) * np.array([s / n for n, s in zip(cells, stretch)])
    i, j, k = (v.ravel() for v in np.meshgrid(*[np.arange(n) for n in cells], indexing="ij"))
    nx, ny = cells[0] + 1, cells[1] + 1
    at = lambda a, b, c: 1 + i + a + nx * (j + b + ny * (k + c))  # noqa: E731
    conn = np.stack([at(0, 0, 0), at(1, 0, 0), at(1, 1, 0), at(0, 1, 0), at(0, 0, 1), at(1, 0, 1), at(1, 1, 1),
                     at(0, 1, 1)], 1)
    if rotate:
        conn = np.stack([c[ORDERS[m % 4]] for m, c in enumerate(conn)])
    low = np.nonzero(np.arange(len(X)) // (nx * ny) == 0)[0] + 1
    return fec.UnstructuredMesh(X, {"b": ("HEX8", conn)}, {"low": low})


def _setup(fec, mesh, fixed=False, **space):
    import torch
    u = fec.VectorFunction(fec.FunctionSpace(mesh, **space), "u")
    asm = fec.SparseMatrixAssembler(u)
    bcs = [fec.DirichletBC(n, lambda X, t: 0.0, nodeset_name="low") for n in u.names] if fixed else []
    p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3), dirichlet_bcs=bcs)
    X = mesh.nodal_coords
    size = np.abs(X).max(0) / max(3, round(len(X) ** (1 / 3)))
    U = X * np.array([0.05, -0.02, 0.03]) + 0.03 * size * np.random.default_rng(9).standard_normal(X.shape)
    U = U.ravel()
    U[asm.dof.dirichlet_dofs - 1] = 0.0
    return asm, p, U, torch.from_numpy(U[asm.dof.unknown_dofs - 1].copy()).cuda()


class environment:
    def __init__(self, **kv):
        self.kv = kv

    def __enter__(self):
        os.environ.update(self.kv)

    def __exit__(self, *exc):
        for k in self.kv:
            del os.environ[k]


@pytest.mark.parametrize("cells, stretch, rotate, fixed, rule", [
    ((2, 1, 1), (1.0, 1.0, 1.0), False, False, "GaussLegendre"),         # (one element alone is a translate of itself)
    ((11, 1, 1), (1.0, 1.0, 1.0), True, False, "GaussLegendre"),        # one element short of a tile
    ((12, 1, 1), (1.0, 1.0, 1.0), False, False, "GaussLegendre"),
    ((13, 1, 1), (1.0, 1.0, 1.0), False, True, "GaussLegendre"),        # one over
    ((5, 6, 7), (1.0, 1.0, 1.0), True, True, "GaussLegendre"),
    ((5, 6, 7), (1.0, 0.02, 0.3), False, False, "GaussLegendre"),       # flat elements
    ((4, 5, 3), (1e-5, 1e-5, 1e-5), False, False, "GaussLegendre"),     # small units
    ((4, 5, 6), (1.0, 1.0, 1.0), False, False, "GaussLobattoLegendre"),
])
def test_matches_oracle(fec, orc, cells, stretch, rotate, fixed, rule):
    import torch
    mesh = _mesh(fec, cells, 4, stretch, rotate)
    asm, p, U, Uu = _setup(fec, mesh, fixed, q_type=rule)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    R, nz = R.cpu().numpy().copy(), K.nzval.cpu().numpy().copy()
    with environment(FEC_HEX8_GENERAL="0"):
        Rp, Kp = fec.assemble_residual_and_stiffness(asm, Uu, p)
        torch.cuda.synchronize()
        Rp, nzp = Rp.cpu().numpy(), Kp.nzval.cpu().numpy()
    assert not np.array_equal(nz, nzp)    # (the two kernels did run)
    assert rel_err(nz, nzp)[2] <= TOL64
    assert max(rel_err(R, Rp)[:2]) <= TOL64
    if rule == "GaussLegendre":           # the oracle's own rule
        args = (blocks_of(mesh), mesh.nodal_coords, "neohookean", p.physics[0].create_properties(), U)
        ab = np.zeros(U.size)
        orc.assemble(*args, want_k=False, abs_out=ab)
        Ro, _, _, nzo = orc.assembled_system(*args, asm.dof.dof_to_unknown, asm.dof.unknown_dofs)
        assert max(rel_err(nz, nzo)) <= TOL64
        assert max(residual_err(R, Ro, ab[asm.dof.unknown_dofs - 1])) <= TOL64


def test_calls_and_workspaces_agree_bitwise(fec):
    import torch
    mesh = _mesh(fec, (7, 5, 6), 2)
    asm, p, _, Uu = _setup(fec, mesh, True)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    with environment(FEC_HEX8_PAIRS="0"):     # node rows of the whole K_e
        R2, K2 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert torch.equal(R2, R) and torch.equal(K2.nzval, nz)
    fec.residual(asm).fill_(float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), R)
    K2.nzval.fill_(float("nan"))
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)


def test_tables_of_another_rule_keep_the_per_element_kernels(fec):
    """Points permuted: not the symmetric rule's order, so nothing changes with the switch."""
    import torch
    mesh = _mesh(fec, (3, 4, 5), 6)
    asm, p, _, Uu = _setup(fec, mesh)
    N, dN, w = asm.reference_tables(1)
    order = [1, 0, 2, 3, 4, 5, 6, 7]
    asm.set_reference_tables([(N[order], dN[order], w[order])])
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    with environment(FEC_HEX8_GENERAL="0"):
        R2, K2 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert torch.equal(R2, R) and torch.equal(K2.nzval, nz)


@pytest.mark.parametrize("cells, stretch, rotate, fixed", [
    ((2, 1, 1), (1.0, 1.0, 1.0), False, False), ((17, 1, 1), (1.0, 1.0, 1.0), True, False),   # one over a CTA's 16
    ((5, 6, 7), (1.0, 0.02, 0.3), True, True), ((4, 5, 3), (1e-5, 1e-5, 1e-5), False, False)])
def test_action_matches_assembled_matrix_and_per_element_kernel(fec, cells, stretch, rotate, fixed):
    import torch
    mesh = _mesh(fec, cells, 8, stretch, rotate)
    asm, p, _, Uu = _setup(fec, mesh, fixed)
    _, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    V = np.random.default_rng(3).standard_normal(asm.dof.unknown_dofs.size)
    Vd = torch.from_numpy(V).cuda()
    A = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Uu, Vd, p).cpu().numpy().copy()
    with environment(FEC_HEX8_GENERAL="0"):
        B = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Uu, Vd, p).cpu().numpy().copy()
    ref = K.to_scipy().T @ V
    scale = abs(K.to_scipy()).T @ np.abs(V)   # the terms of each entry
    assert np.all(np.abs(A - B) <= TOL64 * scale)
    assert np.all(np.abs(A - ref) <= TOL64 * scale)


@pytest.mark.parametrize("phys_name", ["neohookean", "j2"])
def test_action_on_a_skewed_block_of_translates(fec, phys_name):
    """A block of translated parallelepipeds (not boxes): gradients through dxi/dX."""
    import torch
    mesh = fec.StructuredMesh("hex", (0.0,) * 3, (1.0,) * 3, (6, 6, 6))
    X = mesh.nodal_coords @ np.array([[1.0, 0.2, 0.0], [0.1, 0.9, 0.3], [0.0, -0.2, 1.1]])
    mesh = fec.UnstructuredMesh(X, {"b": ("HEX8", mesh.element_conns["block_1"])})
    u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
    asm = fec.SparseMatrixAssembler(u)
    phys = fec.NeoHookean.from_youngs(1.0, 0.3) if phys_name == "neohookean" else fec.J2Plasticity(200.0, 0.3, 0.25, 2.0)
    p = fec.create_parameters(mesh, asm, phys)
    rng = np.random.default_rng(5)
    U = X * np.array([0.004, -0.001, 0.002]) + 1e-4 * rng.standard_normal(X.shape)
    Uu, V = torch.from_numpy(U.ravel()).cuda(), rng.standard_normal(U.size)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    A = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Uu, torch.from_numpy(V).cuda(), p).cpu().numpy()
    M = K.to_scipy()
    assert np.all(np.abs(A - M.T @ V) <= TOL64 * (abs(M).T @ np.abs(V)))
    fused = R.clone()
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), fused)
    with environment(FEC_HEX8_AFFINE="0"):
        R2, K2 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert max(rel_err(fused.cpu().numpy(), R2.cpu().numpy())[:2]) <= TOL64
        assert rel_err(M.data, K2.nzval.cpu().numpy())[2] <= TOL64
