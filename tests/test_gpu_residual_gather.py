"""The residual-only node gather (one thread per node component): bitwise the
residual of the fused residual + tangent assembly, whose gather walks each node
with a warp, over element sizes, several blocks, Dirichlet dofs and nodes with
more adjacent elements than one thread keeps in flight."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(fec, kind):
    from fec_gb300.meshes import box_tet4, box_tet10, merge_meshes
    if kind == "quad4":
        return fec.StructuredMesh("quad", (0.0, 0.0), (1.0, 1.0), (9, 9))
    if kind == "tet4":      # up to 24 elements around a node
        return box_tet4((4, 4, 4))
    if kind == "tet10":
        return box_tet10((3, 3, 3))
    if kind == "blocks":    # two element sizes, one mesh
        return merge_meshes([box_tet4((3, 3, 3)), box_tet10((3, 3, 3))])
    return fec.StructuredMesh("hex", (0.0,) * 3, (1.0,) * 3, (4,) * 3)


@pytest.mark.parametrize("precision", ["fp64", "fp32_element"])
@pytest.mark.parametrize("kind, physics", [("quad4", "poisson"), ("hex8", "poisson"), ("hex8", "neohookean"),
                                           ("hex8", "j2"), ("tet4", "neohookean"), ("tet10", "neohookean"),
                                           ("blocks", "neohookean")])
def test_residual_alone_equals_fused_residual_bitwise(fec, kind, physics, precision):
    import torch
    mesh = _mesh(fec, kind)
    V = fec.FunctionSpace(mesh)
    u = fec.ScalarFunction(V, "u") if physics == "poisson" else fec.VectorFunction(V, "u")
    phys = {"poisson": lambda: fec.Poisson(1.0), "neohookean": lambda: fec.NeoHookean.from_youngs(1.0, 0.3),
            "j2": lambda: fec.J2Plasticity(200.0, 0.3, 0.25, 2.0)}[physics]()
    asm = fec.SparseMatrixAssembler(u, precision=precision)
    bcs = [fec.DirichletBC(u.names[-1], lambda X, t: 0.0, nodeset_name="bottom")] if kind in ("quad4", "hex8") else []
    p = fec.create_parameters(mesh, asm, phys, dirichlet_bcs=bcs)
    rng = np.random.default_rng(3)
    Uu = torch.from_numpy(0.01 * rng.standard_normal(asm.dof.unknown_dofs.size)).cuda()
    R, _ = fec.assemble_residual_and_stiffness(asm, Uu, p)
    fused = R.clone()
    asm.residual_unknowns = torch.full_like(R, float("nan"))
    fec.assemble_vector(asm, fec.residual, Uu, p)
    assert torch.equal(fec.residual(asm), fused)
    assert float(fused.abs().max()) > 0.0
