"""The plan of the gather by output entry belongs to the mesh: it is built at the ninth
assembly that could use it, whatever the Dirichlet conditions were meanwhile, kept when they
change, and gives the per-node gathers' bits with every set of conditions."""
import numpy as np
import pytest

from test_gpu_hex8_general import environment
from test_gpu_pair_gather import _box, _mesh

pytestmark = pytest.mark.gpu


def _assembler(fec, mesh, symbolic):
    ids = np.arange(1, mesh.num_nodes + 1)
    mesh.nodeset_nodes.update({"a": ids[::7], "b": ids[1::5], "c": ids[::11], "all": ids[3:]})
    return fec.SparseMatrixAssembler(fec.VectorFunction(fec.FunctionSpace(mesh), "u"), symbolic=symbolic)


def _parameters(fec, mesh, asm, held):
    bcs = [fec.DirichletBC(v, lambda X, t: 0.0, nodeset_name=s) for v, s in held]
    return fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3), dirichlet_bcs=bcs)


# free, some components of some nodes, whole nodes, all nodes but three
CONDITIONS = [[], [("u_x", "a"), ("u_z", "c")], [(v, "b") for v in ("u_x", "u_y", "u_z")], [],
              [(v, "all") for v in ("u_x", "u_y", "u_z")], [("u_y", "all")]]


@pytest.mark.parametrize("symbolic", ["host", "device"])
@pytest.mark.parametrize("kind", ["box", "part", "one", "sizes", "hex27", "two blocks", "interface", "fan"])
def test_equals_per_node_gathers_bitwise_under_changing_conditions(fec, kind, symbolic):
    import torch
    mesh = _mesh(fec, kind)
    asm = _assembler(fec, mesh, symbolic)
    rng = np.random.default_rng(2)
    for k, held in enumerate(CONDITIONS):
        p = _parameters(fec, mesh, asm, held)
        Uu = torch.from_numpy(1e-3 * rng.standard_normal(asm.dof.unknown_dofs.size)).cuda()
        for _ in range(9 if k == 0 else 1):
            fec.assemble_residual_and_stiffness(asm, Uu, p)
        R, K = fec.residual(asm), fec.stiffness(asm)
        R.fill_(float("nan"))
        K.nzval.fill_(float("nan"))
        fec.assemble_residual_and_stiffness(asm, Uu, p)
        R, nz = R.clone(), K.nzval.clone()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            fec.assemble_residual_and_stiffness(asm, Uu, p)
        K.nzval.fill_(float("nan"))
        graph.replay()
        assert torch.equal(K.nzval, nz)
        with environment(FEC_GATHER_PAIRS="0"):
            R0, K0 = fec.assemble_residual_and_stiffness(asm, Uu, p)
        assert torch.equal(R0, R) and torch.equal(K0.nzval, nz)
        assert bool(torch.isfinite(nz).all()) and bool(torch.isfinite(R).all())


def test_built_at_the_ninth_assembly_and_kept(fec):
    """By the free memory of the device: 262,144 elements' lists and 274,625 nodes' pairs are
    37.7 MB and 74.6 MB."""
    import torch
    mesh = _box(fec, 64)
    asm = _assembler(fec, mesh, "device")
    p = _parameters(fec, mesh, asm, [("u_x", "a")])
    Uu = torch.zeros(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda()
    free = []

    def assemble():
        fec.assemble_residual_and_stiffness(asm, Uu, p)
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])

    for k in range(12):
        if k == 5:     # new conditions do not start the count again
            p = _parameters(fec, mesh, asm, [("u_y", "a")])
            Uu = torch.zeros(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda()
        assemble()
    used = -np.diff(free) / 1e6
    pairs = (193 ** 3 + 65 ** 3) // 2 * 20e-6
    assert abs(used[7] - (pairs + 64 ** 3 * 36 * 4e-6)) <= 6    # (the allocator's granularity)
    assert np.abs(used[[0, 1, 2, 3, 5, 6, 8, 9, 10]]).max() <= 1
    p = _parameters(fec, mesh, asm, [("u_z", "b")])
    Uu = torch.zeros(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda()
    assemble()
    kept = free[-1]
    assemble()
    assert free[-1] == kept
