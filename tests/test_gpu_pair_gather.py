"""The gather of symmetric-half element matrices by output entry against the
per-node gathers, bitwise: boxes, distorted meshes, Dirichlet dofs on parts of the
nodes, several element sizes, blocks that share nodes, nodes of many elements."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(fec, n, move=0.0):
    mesh = fec.StructuredMesh("hex", (0.0,) * 3, (1.0,) * 3, (n + 1,) * 3)
    X = mesh.nodal_coords + move / n * np.random.default_rng(1).uniform(-1, 1, mesh.nodal_coords.shape)
    return fec.UnstructuredMesh(X, {"b": ("HEX8", mesh.element_conns["block_1"])}, mesh.nodeset_nodes)


def _mesh(fec, kind):
    from fec_gb300.meshes import box_hex27, box_tet4, box_tet10, merge_meshes
    if kind == "box":
        return _box(fec, 6)
    if kind == "part":
        return _box(fec, 5, 0.15)
    if kind == "one":
        return _box(fec, 1)
    if kind == "sizes":          # disjoint blocks of four sizes
        return merge_meshes([box_tet4((4, 4, 4)), box_tet10((3, 3, 3)), box_hex27((3, 4, 3)), _box(fec, 3)])
    if kind == "hex27":
        return box_hex27((4, 3, 4))
    if kind == "two blocks":     # one element size, a shared face
        m = _box(fec, 4)
        c = m.element_conns["b"]
        return fec.UnstructuredMesh(m.nodal_coords, {"a": ("HEX8", c[:30]), "b": ("HEX8", c[30:])}, m.nodeset_nodes)
    if kind == "interface":      # hex8 and tet4 blocks sharing the nodes of a face
        m = _box(fec, 4)
        c = m.element_conns["b"]
        k = np.array([[0, 1, 2, 6], [0, 2, 3, 6], [0, 3, 7, 6], [0, 7, 4, 6], [0, 4, 5, 6], [0, 5, 1, 6]])
        return fec.UnstructuredMesh(m.nodal_coords, {"h": ("HEX8", c[:32]), "t": ("TETRA4", c[32:][:, k].reshape(-1, 4))},
                                    m.nodeset_nodes)
    # a fan of 20 hexes around one edge: 20 elements at its two nodes
    n = 20
    t = 2 * np.pi * np.arange(2 * n) / (2 * n)
    ring = np.stack([np.cos(t), np.sin(t)], 1)
    X = np.concatenate([np.c_[np.vstack([[0.0, 0.0], ring]), np.full(2 * n + 1, z)] for z in (0.0, 1.0)])
    lo = [[1, 2 + 2 * i, 3 + 2 * i, 2 + (2 * i + 2) % (2 * n)] for i in range(n)]
    conn = np.array([q + [v + 2 * n + 1 for v in q] for q in lo])
    return fec.UnstructuredMesh(X, {"b": ("HEX8", conn)}, {})


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("kind", ["box", "part", "one", "sizes", "hex27", "two blocks", "interface", "fan"])
def test_equals_per_node_gathers_bitwise(fec, kind, fixed):
    import torch
    mesh = _mesh(fec, kind)
    u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
    asm = fec.SparseMatrixAssembler(u)
    sets = mesh.nodeset_nodes
    if fixed and not sets:
        ids = np.arange(1, mesh.num_nodes + 1)
        sets = {"left": ids[::7], "bottom": ids[1::5], "back": ids[::11]}
        mesh.nodeset_nodes.update(sets)
    bcs = [fec.DirichletBC(v, lambda X, t: 0.0, nodeset_name=f)
           for f, vs in (("left", u.names), ("bottom", u.names[:1]), ("back", u.names[1:])) for v in vs] if fixed else []
    p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3), dirichlet_bcs=bcs)
    rng = np.random.default_rng(2)
    Uu = torch.from_numpy(1e-3 * rng.standard_normal(asm.dof.unknown_dofs.size)).cuda()
    out = []
    for switch in (None, "0"):
        if switch:
            os.environ["FEC_GATHER_PAIRS"] = switch
        try:
            R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
            K.nzval.fill_(float("nan"))
            R.fill_(float("nan"))
            R, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
            out.append((R.clone(), K.nzval.clone()))
            K.nzval.fill_(float("nan"))
            fec.assemble_stiffness(asm, fec.stiffness, Uu, p)
            assert torch.equal(fec.stiffness(asm).nzval, out[-1][1])
        finally:
            os.environ.pop("FEC_GATHER_PAIRS", None)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert bool(torch.isfinite(out[0][1]).all()) and bool(torch.isfinite(out[0][0]).all())


def test_new_dirichlet_conditions_renew_the_plan_and_capture_works_without_one(fec):
    import torch
    mesh = _box(fec, 4, 0.1)
    u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
    asm = fec.SparseMatrixAssembler(u)
    phys = fec.NeoHookean.from_youngs(1.0, 0.3)
    for faces in (["left"], ["left", "top"], []):
        p = fec.create_parameters(mesh, asm, phys,
                                  dirichlet_bcs=[fec.DirichletBC("u_x", lambda X, t: 0.0, nodeset_name=f) for f in faces])
        Uu = 1e-3 * torch.randn(asm.dof.unknown_dofs.size, dtype=torch.float64, device="cuda")
        os.environ["FEC_GATHER_PAIRS"] = "0"   # allocations, without a plan
        try:
            _, K = fec.assemble_residual_and_stiffness(asm, Uu, p)
        finally:
            del os.environ["FEC_GATHER_PAIRS"]
        ref = K.nzval.clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):          # the first use of the plan's rule is under capture
            fec.assemble_residual_and_stiffness(asm, Uu, p)
        K.nzval.fill_(float("nan"))
        graph.replay()
        assert torch.equal(K.nzval, ref)
        K.nzval.fill_(float("nan"))
        fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert torch.equal(K.nzval, ref)
