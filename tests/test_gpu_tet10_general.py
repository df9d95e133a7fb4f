"""FP64 Neo-Hookean tet10 blocks of any shape on the tensor cores against the CPU oracle
and the other kernels: edges of the tiles (12 and 24 elements), straight, curved, flat and
small elements, permuted local numberings, translation classes, Dirichlet dofs, and the
calls that must agree bitwise."""
import numpy as np
import pytest

from helpers import blocks_of, rel_err, residual_err
from test_gpu_hex8_general import TOL64, _setup, environment

pytestmark = pytest.mark.gpu
TETS = ((0, 1, 3, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7), (0, 4, 5, 7), (0, 5, 1, 7))  # corner bits x, y, z
EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))
TURN = ([0, 1, 2, 3], [1, 2, 0, 3], [2, 0, 1, 3], [1, 0, 3, 2])     # rotations of a tet


def _mesh(fec, cells, count, bend=0.0, move=0.1, stretch=(1.0, 1.0, 1.0), rotate=False):
    n = 2 * np.array(cells) + 1
    ids = np.arange(n.prod()).reshape(n[::-1])
    X = np.stack([v.ravel() for v in np.meshgrid(*[np.arange(m) for m in n[::-1]], indexing="ij")][::-1], 1) * 1.0
    rng = np.random.default_rng(8)
    X += move * 2 * rng.uniform(-1, 1, X.shape)
    conn = []
    for k, j, i in np.ndindex(*cells[::-1]):
        for t, tet in enumerate(TETS):
            c = np.array([[2 * i + 2 * (v & 1), 2 * j + (v & 2), 2 * k + (v & 4) // 2] for v in tet])
            if rotate:
                c = c[TURN[(t + i) % 4]]
            p = np.concatenate([c, [(c[a] + c[b]) // 2 for a, b in EDGES]])
            conn.append(ids[p[:, 2], p[:, 1], p[:, 0]])
    conn = np.array(conn)[:count]
    if move:
        for e, (a, b) in enumerate(EDGES):
            X[conn[:, 4 + e]] = 0.5 * (X[conn[:, a]] + X[conn[:, b]])
    X += bend * 2 * rng.uniform(-1, 1, X.shape)
    used, conn = np.unique(conn, return_inverse=True)
    X = X[used] * 0.5 * np.array(stretch) / max(cells)
    low = np.nonzero(X[:, 2] < 0.3 * stretch[2] / max(cells))[0] + 1
    return fec.UnstructuredMesh(X, {"b": ("TETRA10", conn.reshape(-1, 10) + 1)}, {"low": low})


@pytest.mark.parametrize("cells, count, kw", [
    ((1, 1, 1), 1, {}), ((1, 1, 2), 11, {}), ((2, 1, 1), 12, {}), ((3, 1, 1), 13, dict(bend=0.04)),
    ((2, 2, 1), 24, dict(bend=0.04)), ((5, 1, 1), 25, dict(rotate=True)),
    ((4, 5, 3), 360, dict(bend=0.04, rotate=True)),
    ((4, 5, 3), 347, dict(stretch=(1.0, 0.03, 0.3))),        # flat elements
    ((3, 4, 5), 360, dict(stretch=(1e-5,) * 3, bend=0.04)),  # small units
    ((4, 4, 4), 384, dict(move=0.0)),                        # translation classes
])
@pytest.mark.parametrize("fixed", [False, True])
def test_matches_oracle(fec, orc, cells, count, kw, fixed):
    import torch
    mesh = _mesh(fec, cells, count, **kw)
    asm, p, U, Uu = _setup(fec, mesh, fixed)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    R, nz = R.cpu().numpy().copy(), K.nzval.cpu().numpy().copy()
    with environment(FEC_TET10_GENERAL="0"):
        Rp, Kp = fec.assemble_residual_and_stiffness(asm, Uu, p)
        torch.cuda.synchronize()
        Rp, nzp = Rp.cpu().numpy(), Kp.nzval.cpu().numpy()
    assert not np.array_equal(nz, nzp)    # (the two kernels did run)
    assert rel_err(nz, nzp)[2] <= TOL64
    args = (blocks_of(mesh), mesh.nodal_coords, "neohookean", p.physics[0].create_properties(), U)
    ab = np.zeros(U.size)
    orc.assemble(*args, want_k=False, abs_out=ab)
    Ro, _, _, nzo = orc.assembled_system(*args, asm.dof.dof_to_unknown, asm.dof.unknown_dofs)
    assert max(rel_err(nz, nzo)) <= TOL64
    assert max(residual_err(R, Ro, ab[asm.dof.unknown_dofs - 1])) <= TOL64


def test_calls_agree_bitwise_and_other_rules_keep_their_kernels(fec):
    import torch
    mesh = _mesh(fec, (3, 4, 5), 360, bend=0.04)
    asm, p, _, Uu = _setup(fec, mesh, True)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    fec.residual(asm).fill_(float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), R)
    K.nzval.fill_(float("nan"))
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)
    N, dN, w = asm.reference_tables(1)
    order = [2, 0, 3, 1]                  # the points in another order: the same rule
    asm.set_reference_tables([(N[order], dN[order], w[order])])
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)
    asm.set_reference_tables([(N, dN * (1 + 1e-9), w)])   # not its gradients any more
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    other = fec.stiffness(asm).nzval.clone()
    with environment(FEC_TET10_GENERAL="0"):
        fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
        assert torch.equal(fec.stiffness(asm).nzval, other)
