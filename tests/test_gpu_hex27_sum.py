"""FP64 Neo-Hookean hex27 blocks by sum factorisation against the CPU oracle and the
per-element kernel: one element up to several per CTA, straight, curved, flat and small
elements, permuted local numberings, translation classes, Dirichlet dofs, Lobatto points,
both workspaces, and the calls that must agree bitwise."""
import numpy as np
import pytest

from helpers import blocks_of, rel_err, residual_err
from test_gpu_hex8_general import TOL64, _setup, environment

pytestmark = pytest.mark.gpu


def _mesh(fec, cells, bend=0.0, stretch=(1.0, 1.0, 1.0), rotate=False):
    n = 2 * np.array(cells) + 1
    ids = np.arange(n.prod()).reshape(n[::-1])
    X = np.stack([v.ravel() for v in np.meshgrid(*[np.arange(m) for m in n[::-1]], indexing="ij")][::-1], 1) * 1.0
    X += bend * np.random.default_rng(8).uniform(-1, 1, X.shape)
    conn = []
    for k, j, i in np.ndindex(*cells[::-1]):
        c = ids[2 * k:2 * k + 3, 2 * j:2 * j + 3, 2 * i:2 * i + 3]   # [z][y][x]
        if rotate:                                                  # about z, or x -> y -> z -> x
            c = (c, c.transpose(0, 2, 1)[:, :, ::-1], c.transpose(1, 2, 0), c[:, ::-1, ::-1])[(i + j) % 4]
        conn.append(c.ravel())
    X = X * 0.5 * np.array(stretch) / max(cells)
    low = np.nonzero(X[:, 2] < 0.3 * stretch[2] / max(cells))[0] + 1
    return fec.UnstructuredMesh(X, {"b": ("HEX27", np.array(conn) + 1)}, {"low": low})


@pytest.mark.parametrize("cells, kw, rule", [
    ((1, 1, 1), dict(bend=0.15), "GaussLegendre"), ((2, 1, 1), dict(bend=0.15), "GaussLegendre"),
    ((3, 2, 2), dict(bend=0.15, rotate=True), "GaussLegendre"),
    ((10, 10, 10), dict(bend=0.15, rotate=True), "GaussLegendre"),   # three elements a CTA, some with two
    ((3, 2, 3), dict(bend=0.15, stretch=(1.0, 0.03, 0.3)), "GaussLegendre"),
    ((3, 2, 2), dict(bend=0.15, stretch=(1e-5,) * 3), "GaussLegendre"),
    ((3, 4, 3), dict(), "GaussLegendre"),                            # one translation class
    ((3, 2, 2), dict(bend=0.15), "GaussLobattoLegendre"),
])
@pytest.mark.parametrize("fixed", [False, True])
def test_matches_oracle(fec, orc, cells, kw, rule, fixed):
    import torch
    mesh = _mesh(fec, cells, **kw)
    asm, p, U, Uu = _setup(fec, mesh, fixed, q_type=rule)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    R, nz = R.cpu().numpy().copy(), K.nzval.cpu().numpy().copy()
    with environment(FEC_HEX27_GENERAL="0"):
        Rp, Kp = fec.assemble_residual_and_stiffness(asm, Uu, p)
        torch.cuda.synchronize()
        Rp, nzp = Rp.cpu().numpy(), Kp.nzval.cpu().numpy()
    assert not np.array_equal(nz, nzp)    # (the two kernels did run)
    assert rel_err(nz, nzp)[2] <= TOL64
    assert max(rel_err(R, Rp)[:2]) <= TOL64
    if rule == "GaussLegendre":
        args = (blocks_of(mesh), mesh.nodal_coords, "neohookean", p.physics[0].create_properties(), U)
        ab = np.zeros(U.size)
        orc.assemble(*args, want_k=False, abs_out=ab)
        Ro, _, _, nzo = orc.assembled_system(*args, asm.dof.dof_to_unknown, asm.dof.unknown_dofs)
        assert max(rel_err(nz, nzo)) <= TOL64
        assert max(residual_err(R, Ro, ab[asm.dof.unknown_dofs - 1])) <= TOL64


def test_calls_and_workspaces_agree_bitwise(fec):
    import torch
    mesh = _mesh(fec, (4, 3, 5), bend=0.15, rotate=True)
    asm, p, _, Uu = _setup(fec, mesh, True)
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    with environment(FEC_HEX27_PAIRS="0"):     # whole matrices
        R2, K2 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert torch.equal(R2, R) and torch.equal(K2.nzval, nz)
    fec.residual(asm).fill_(float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), R)
    K.nzval.fill_(float("nan"))
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.stiffness(asm).nzval, nz)


def test_other_point_orders_keep_the_per_element_kernel(fec):
    import torch
    mesh = _mesh(fec, (2, 2, 1), bend=0.15)
    asm, p, _, Uu = _setup(fec, mesh)
    N, dN, w = asm.reference_tables(1)
    order = [1, 0, *range(2, 27)]
    asm.set_reference_tables([(N[order], dN[order], w[order])])
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    nz = fec.stiffness(asm).nzval.clone()
    with environment(FEC_HEX27_GENERAL="0"):
        fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
        assert torch.equal(fec.stiffness(asm).nzval, nz)
