"""FP64 Poisson kernels at the edges of their launch shapes against the oracle: the
small and the large CTA of quad4 and hex8, blocks of translated boxes (shared sines)
and of skewed translates, partial last CTAs; residual and tangent alone bitwise the
fused pass's; one launch for the field update with a Dirichlet dof that is an unknown."""
import numpy as np
import pytest

from helpers import blocks_of, rel_err

pytestmark = pytest.mark.gpu
SKEW = np.array([[1.0, 0.2, 0.0], [0.1, 0.9, 0.3], [0.0, -0.2, 1.1]])


# quad4: 9 elements (a CTA of 8 and one), 10,000 (CTAs of 64); hex8: 1, 27, 17^3 in CTAs of 16
@pytest.mark.parametrize("kind, n, shape", [("quad", 3, "box"), ("quad", 100, "box"), ("quad", 7, "bent"),
                                            ("hex", 1, "box"), ("hex", 3, "box"), ("hex", 17, "box"), ("hex", 3, "skew"),
                                            ("hex", 3, "bent"), ("hex", 14, "bent")])
def test_matches_oracle(fec, orc, kind, n, shape):
    import torch
    dim = 2 if kind == "quad" else 3
    mesh = fec.StructuredMesh(kind, (0.0,) * dim, (1.0,) * dim, (n + 1,) * dim)
    X = mesh.nodal_coords
    if shape == "skew":
        X = X @ SKEW
    if shape == "bent":
        X = X + 0.2 / n * np.random.default_rng(1).uniform(-1, 1, X.shape)
    mesh = fec.UnstructuredMesh(X, {"b": ({"quad": "QUAD4", "hex": "HEX8"}[kind], mesh.element_conns["block_1"])},
                                mesh.nodeset_nodes)
    u = fec.ScalarFunction(fec.FunctionSpace(mesh), "u")
    asm = fec.SparseMatrixAssembler(u)
    p = fec.create_parameters(mesh, asm, fec.Poisson(1.5),
                              dirichlet_bcs=[fec.DirichletBC("u", lambda x, t: 0.0, nodeset_name="bottom")])
    U = np.random.default_rng(2).uniform(-1.0, 1.0, mesh.num_nodes)
    U[asm.dof.dirichlet_dofs - 1] = 0.0
    Uu = torch.from_numpy(U[asm.dof.unknown_dofs - 1].copy()).cuda()
    R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
    R, nz = R.clone(), K.nzval.clone()
    Ro, _, _, nzo = orc.assembled_system(blocks_of(mesh), X, "poisson", [1.5], U, asm.dof.dof_to_unknown,
                                         asm.dof.unknown_dofs)
    assert max(rel_err(nz.cpu().numpy(), nzo)) <= 1e-12
    assert max(rel_err(R.cpu().numpy(), Ro)[:2]) <= 1e-12
    fec.assemble_vector(asm, fec.residual, Uu, p)
    fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
    assert torch.equal(fec.residual(asm), R) and torch.equal(fec.stiffness(asm).nzval, nz)


def test_field_update_order(fec):
    """Dirichlet values first, then the unknowns: an unknown dof keeps its unknown."""
    import ctypes as C
    import torch
    from fec_gb300 import _lib
    mesh = fec.StructuredMesh("quad", (0.0, 0.0), (1.0, 1.0), (5, 5))
    asm = fec.SparseMatrixAssembler(fec.ScalarFunction(fec.FunctionSpace(mesh), "u"))
    p = fec.create_parameters(mesh, asm, fec.Poisson(1.0),
                              dirichlet_bcs=[fec.DirichletBC("u", lambda x, t: 0.0, nodeset_name="bottom")])
    n = asm.dof.unknown_dofs.size
    Uu = torch.arange(1, n + 1, dtype=torch.float64).cuda()
    dofs = torch.arange(1, 26, dtype=torch.int64).cuda()      # every dof, unknowns too
    vals = -torch.arange(1, 26, dtype=torch.float64).cuda()
    asm._call("fec_update_field", _lib.ptr(p.field), _lib.ptr(Uu), 25, _lib.ptr(dofs), _lib.ptr(vals),
              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    want = -np.arange(1, 26, dtype=float)
    want[asm.dof.unknown_dofs - 1] = np.arange(1, n + 1)
    assert np.array_equal(p.field.cpu().numpy(), want)
