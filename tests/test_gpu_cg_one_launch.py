"""The conjugate-gradient solve in one cooperative launch against the three kernels an
iteration, on both sides of its size rule: one to four rows per thread, a CTA whose
entries do not fit its shared memory, iteration limits, Jacobi."""
import os

import numpy as np
import pytest

from test_gpu_cg_kernels import _solve, _system

pytestmark = pytest.mark.gpu


def _both(asm, K, max_iter, rtol, jacobi):
    import torch
    n = asm.dof.unknown_dofs.size
    rng = np.random.default_rng(n)
    b, x0 = torch.from_numpy(rng.standard_normal(n)).cuda(), torch.from_numpy(rng.standard_normal(n)).cuda()
    out = []
    for switch in (None, "0"):
        if switch:
            os.environ["FEC_CG_COOP"] = switch
        try:
            x = x0.clone()
            it, rr = _solve(asm, K, b, x, max_iter, rtol, jacobi)
            again = x0.clone()
            it2, rr2 = _solve(asm, K, b, again, max_iter, rtol, jacobi)
            assert it2 == it and np.array_equal(rr, rr2, equal_nan=True) and torch.equal(x.nan_to_num(), again.nan_to_num())
            out.append((it, rr, x))
        finally:
            os.environ.pop("FEC_CG_COOP", None)
    return out


# rows per CTA: 1; 17; 256; 264 (two a thread); 945 (four); beyond the rule
@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("cells, inside", [(2, True), (5, True), (17, True), (201, True), (380, True), (420, False)])
def test_same_iterations(fec, cells, inside, jacobi):
    import torch
    asm, K = _system(fec, "quad4", (cells,))
    (it, rr, x), (it0, rr0, x0) = _both(asm, K, 23, 0.0, jacobi)
    assert it == it0 == 23
    if not inside:
        assert torch.equal(x, x0) and rr == rr0
    if np.isnan(rr0):    # one unknown: 0 / 0 once its residual is zero
        assert np.isnan(rr) and torch.equal(x.isnan(), x0.isnan())
        return
    # rounding of 23 iterations (sums in another order), with room for its growth
    assert float((x - x0).norm()) <= 1e-9 * float(x0.norm())
    assert abs(rr - rr0) <= 1e-9 + 1e-6 * rr0


def test_long_rows_of_one_cta(fec):
    """Hex27 rows after the rows of many tet4 elements: the last CTAs have more entries than
    fit their shared memory."""
    import torch
    from fec_gb300.meshes import box_hex27, box_tet4, merge_meshes
    mesh = merge_meshes([box_tet4((22, 22, 22)), box_hex27((5, 5, 5))])
    u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
    ids = np.arange(1, mesh.num_nodes + 1)
    mesh.nodeset_nodes["low"] = ids[mesh.nodal_coords[:, 2] < 1e-9]
    asm = fec.SparseMatrixAssembler(u)
    bcs = [fec.DirichletBC(v, lambda X, t: 0.0, nodeset_name="low") for v in u.names]
    p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3), dirichlet_bcs=bcs)
    n = asm.dof.unknown_dofs.size
    _, K = fec.assemble_residual_and_stiffness(asm, torch.zeros(n, dtype=torch.float64).cuda(), p)
    lengths = np.diff(K.to_scipy().indptr)
    grid = min(torch.cuda.get_device_properties(0).multi_processor_count, max(-(-n // 256), int(lengths.sum()) // 14742 + 1))
    rows = -(-n // grid)
    per_cta = np.add.reduceat(lengths, np.arange(0, n, rows))
    assert per_cta.max() > 16384 > per_cta.min() and lengths.sum() <= grid * 16384
    (it, rr, x), (it0, rr0, x0) = _both(asm, K, 23, 0.0, True)
    assert it == it0 == 23 and float((x - x0).norm()) <= 1e-9 * float(x0.norm())
