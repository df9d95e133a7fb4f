"""The plan of the gather by output entry belongs to the mesh: it is built after some assemblies
that could have used it (the fifth on a large mesh; the first with FEC_GATHER_PAIRS=1),
whatever the Dirichlet conditions were meanwhile, kept when they change, and gives the
per-node gathers' bits with every set of conditions."""
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
        with environment(FEC_GATHER_PAIRS="1"):
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


@pytest.mark.parametrize("n, built", [(64, 5), (12, None)])
def test_built_when_it_has_paid_for_itself_and_kept(fec, n, built):
    """By the free memory of the device: the lists of 64^3 elements and the pairs of 65^3 nodes
    are 37.7 MB and 74.6 MB; 12^3 elements (62,208 pairs) wait for 68 assemblies."""
    import torch
    mesh = _box(fec, n)
    asm = _assembler(fec, mesh, "device")
    free = []

    def assemble(held, count=1):
        p = _parameters(fec, mesh, asm, held)
        Uu = torch.zeros(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda()
        for _ in range(count):
            fec.assemble_residual_and_stiffness(asm, Uu, p)
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])

    assemble([("u_x", "a")], 2)
    assemble([("u_y", "a")], 8)      # new conditions do not start the count again
    used = -np.diff(free) / 1e6      # used[k]: by assembly k + 2
    size = ((3 * n + 1) ** 3 + (n + 1) ** 3) // 2 * 20e-6 + n ** 3 * 36 * 4e-6
    for k, u in enumerate(used, start=2):
        if k == built:
            assert abs(u - size) <= 6    # (the allocator's granularity)
        elif k != 3:                     # (the third has new conditions: other arrays)
            assert abs(u) <= 1
    assemble([("u_z", "b")], 2)
    assert free[-1] == free[-2]
