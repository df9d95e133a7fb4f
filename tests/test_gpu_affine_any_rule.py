"""FP64 blocks of translated hex8 elements with 8-point tables that are not a symmetric rule's
(points in another order, points and weights of no symmetry): the tensor-core kernel against
the oracle with the same tables and the per-element kernels, tile edges and skewed elements,
the calls that must agree bitwise, and the workspace of the symmetric half."""
import numpy as np
import pytest

from helpers import blocks_of, rel_err, residual_err
from test_gpu_hex8_general import TOL64, environment
from test_zz_no_alloc import _noalloc

pytestmark = pytest.mark.gpu
NODES = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]])


def _tables(kind):
    t = 1 / np.sqrt(3.0)
    x = t * (2 * np.array([[i & 1, i >> 1 & 1, i >> 2] for i in range(8)]) - 1.0)
    w = np.ones(8)
    if kind == "permuted":
        order = [1, 0, 2, 7, 4, 6, 5, 3]
        x = x[order]
    else:
        rng = np.random.default_rng(3)
        x, w = 0.9 * x + 0.1 * rng.uniform(-1, 1, x.shape), rng.uniform(0.8, 1.2, 8)
    f = (1 + x[:, None, :] * NODES) / 2
    dN = np.stack([NODES[:, j] / 2 * f[:, :, (j + 1) % 3] * f[:, :, (j + 2) % 3] for j in range(3)], 2)
    return f.prod(2), dN, w


def _problem(fec, nodes, phys_name, kind, skew):
    import torch
    z, y, x = (v.ravel() for v in np.meshgrid(*[np.arange(n) for n in nodes[::-1]], indexing="ij"))
    first = ((x < nodes[0] - 1) & (y < nodes[1] - 1) & (z < nodes[2] - 1)).nonzero()[0]
    dx, dy, dz = 1, nodes[0], nodes[0] * nodes[1]
    conn = first[:, None] + 1 + np.array([0, dx, dx + dy, dy, dz, dx + dz, dx + dy + dz, dy + dz])
    X = np.stack([x, y, z], 1) * 0.0625     # (exact coordinates: translates of one another)
    if skew:
        X = X @ np.array([[1.0, 0.25, 0.0], [0.125, 0.875, 0.25], [0.0, -0.25, 1.125]])
    mesh = fec.UnstructuredMesh(X, {"b": ("HEX8", conn)})
    asm = fec.SparseMatrixAssembler(fec.VectorFunction(fec.FunctionSpace(mesh), "u"))
    tables = _tables(kind)
    asm.set_reference_tables([tables])
    phys = fec.NeoHookean.from_youngs(1.0, 0.3) if phys_name == "neohookean" else fec.J2Plasticity(200.0, 0.3, 0.25, 2.0)
    p = fec.create_parameters(mesh, asm, phys)
    X = mesh.nodal_coords
    U = X * np.array([0.004, -0.001, 0.002]) + 1e-4 * 0.0625 * np.random.default_rng(5).standard_normal(X.shape)
    return mesh, asm, p, tables, U.ravel(), torch.from_numpy(U.ravel().copy()).cuda()


@pytest.mark.parametrize("phys_name", ["neohookean", "j2"])
@pytest.mark.parametrize("kind", ["permuted", "asymmetric"])
@pytest.mark.parametrize("nodes, skew", [((2, 2, 2), False), ((13, 2, 2), True), ((14, 2, 2), False), ((6, 7, 5), True)])
def test_matches_oracle_and_per_element_kernels(fec, orc, nodes, skew, kind, phys_name):
    import torch
    mesh, asm, p, tables, U, Uu = _problem(fec, nodes, phys_name, kind, skew)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz, state = R.clone(), K.nzval.clone(), p.state_new.clone() if phys_name == "j2" else None
    Rd, nzd = R.cpu().numpy(), nz.cpu().numpy()
    fec.residual(asm).fill_(float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), R)
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)
    V = torch.from_numpy(np.random.default_rng(1).standard_normal(U.size)).cuda()
    A = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Uu, V, p).cpu().numpy()
    M = K.to_scipy()
    assert np.all(np.abs(A - M.T @ V.cpu().numpy()) <= TOL64 * (abs(M).T @ np.abs(V.cpu().numpy())))
    with environment(FEC_HEX8_AFFINE="0"):
        R2, K2 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert not torch.equal(K2.nzval, nz)      # (the two kernels did run)
        assert rel_err(nzd, K2.nzval.cpu().numpy())[2] <= TOL64
        assert max(rel_err(Rd, R2.cpu().numpy())[:2]) <= TOL64
    so = p.state_old.cpu().numpy() if state is not None else None
    sn = np.zeros_like(so) if state is not None else None
    with orc.reference_tables("HEX8", *tables):
        args = (blocks_of(mesh), mesh.nodal_coords, phys_name, p.physics[0].create_properties(), U)
        Ro, _, _, nzo = orc.assembled_system(*args, asm.dof.dof_to_unknown, asm.dof.unknown_dofs, so, sn)
    assert max(rel_err(nzd, nzo)) <= TOL64
    assert max(rel_err(Rd, Ro)[:2]) <= TOL64
    if state is not None:
        assert np.abs(state.cpu().numpy().ravel() - sn.ravel()).max() <= TOL64


@pytest.mark.parametrize("phys_name", ["neohookean", "j2"])
def test_workspace_is_the_symmetric_half(fec, phys_name):
    """15,625 elements: the symmetric halves fit the static workspace, whole matrices do not."""
    mesh, asm, p, _, _, Uu = _problem(fec, (26, 26, 26), phys_name, "permuted", False)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.cpu().numpy().copy(), K.nzval.cpu().numpy().copy()
    R2, nz2, _ = _noalloc(fec, asm, p, 0)
    assert np.array_equal(R, R2) and np.array_equal(nz, nz2)
