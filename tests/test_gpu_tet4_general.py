"""FP64 Neo-Hookean tet4 blocks against the CPU oracle and the per-element kernel: edges of
the 64-element blocks, moved nodes, flat and small elements, permuted local numberings,
Dirichlet dofs, and the calls that must agree bitwise."""
import numpy as np
import pytest

from helpers import blocks_of, rel_err, residual_err
from test_gpu_hex8_general import TOL64, _setup, environment
from test_gpu_tet10_general import TETS, TURN

pytestmark = pytest.mark.gpu


def _mesh(fec, cells, count, stretch=(1.0, 1.0, 1.0), rotate=False):
    n = np.array(cells) + 1
    ids = np.arange(n.prod()).reshape(n[::-1])
    X = np.stack([v.ravel() for v in np.meshgrid(*[np.arange(m) for m in n[::-1]], indexing="ij")][::-1], 1) * 1.0
    X += np.random.default_rng(8).uniform(-0.1, 0.1, X.shape)
    conn = []
    for k, j, i in np.ndindex(*cells[::-1]):
        for t, tet in enumerate(TETS):
            c = np.array([ids[k + (v >> 2 & 1), j + (v >> 1 & 1), i + (v & 1)] for v in tet])
            conn.append(c[TURN[(t + i) % 4]] if rotate else c)
    used, conn = np.unique(np.array(conn)[:count], return_inverse=True)
    X = X[used] * np.array(stretch) / max(cells)
    low = np.nonzero(X[:, 2] < 0.3 * stretch[2] / max(cells))[0] + 1
    return fec.UnstructuredMesh(X, {"b": ("TETRA4", conn.reshape(-1, 4) + 1)}, {"low": low})


@pytest.mark.parametrize("cells, count, kw", [
    ((1, 1, 1), 1, {}), ((3, 2, 2), 63, {}), ((3, 2, 2), 64, dict(rotate=True)), ((3, 2, 2), 65, {}),
    ((5, 4, 6), 720, dict(rotate=True)),
    ((5, 4, 6), 720, dict(stretch=(1.0, 0.03, 0.3))),
    ((4, 4, 4), 384, dict(stretch=(1e-5,) * 3)),
])
@pytest.mark.parametrize("fixed", [False, True])
def test_matches_oracle(fec, orc, cells, count, kw, fixed):
    import torch
    mesh = _mesh(fec, cells, count, **kw)
    asm, p, U, Uu = _setup(fec, mesh, fixed)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    R, nz = R.cpu().numpy().copy(), K.nzval.cpu().numpy().copy()
    with environment(FEC_TET4_GENERAL="0"):
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


def test_calls_agree_bitwise(fec):
    import torch
    mesh = _mesh(fec, (5, 4, 6), 700)
    asm, p, _, Uu = _setup(fec, mesh, True)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    fec.residual(asm).fill_(float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), R)
    K.nzval.fill_(float("nan"))
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)


def test_block_after_one_of_odd_size(fec, orc):
    """27 node numbers before the block's: its connectivity is not 16-byte aligned."""
    import torch
    from fec_gb300.meshes import box_hex27, merge_meshes
    t = _mesh(fec, (3, 2, 2), 70)
    mesh = merge_meshes([box_hex27((2, 2, 2)), t])
    asm, p, U, Uu = _setup(fec, mesh)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    args = (blocks_of(mesh), mesh.nodal_coords, "neohookean", p.physics[0].create_properties(), U)
    Ro, _, _, nzo = orc.assembled_system(*args, asm.dof.dof_to_unknown, asm.dof.unknown_dofs)
    assert max(rel_err(K.nzval.cpu().numpy(), nzo)) <= TOL64
    assert max(rel_err(R.cpu().numpy(), Ro)[:2]) <= TOL64
