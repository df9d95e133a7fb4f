"""FP64 Neo-Hookean tet4: errors of residual and tangent against the same sums in extended
precision are no larger than the per-element kernel's.  Root mean squares over six meshes of
750 elements: some 3,900 residual values, so two equal errors differ by about a per cent."""
import numpy as np
import pytest

from test_gpu_flat_elements import LD, _exact
from test_gpu_hex8_general import environment

pytestmark = pytest.mark.gpu
TETS = ((0, 1, 3, 7), (0, 3, 2, 7), (0, 2, 6, 7), (0, 6, 4, 7), (0, 4, 5, 7), (0, 5, 1, 7))  # corner bits x, y, z


def _mesh(fec, n, seed):
    ids = np.arange((n + 1) ** 3).reshape((n + 1,) * 3)
    z, y, x = np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij")
    X = np.stack([x.ravel(), y.ravel(), z.ravel()], 1) / n
    X = X + np.random.default_rng(seed).uniform(-0.15, 0.15, X.shape) / n
    conn = [[ids[k + (v >> 2), j + (v >> 1 & 1), i + (v & 1)] for v in tet]
            for k, j, i in np.ndindex(n, n, n) for tet in TETS]
    return fec.UnstructuredMesh(X, {"b": ("TETRA4", np.array(conn) + 1)})


@pytest.mark.parametrize("strain", [1e-6, 1e-3, 0.05])
def test_errors_are_no_larger_than_the_per_element_kernels(fec, strain):
    import torch
    dN, w = np.concatenate([-np.ones((1, 3), LD), np.eye(3, dtype=LD)])[None], [LD(1) / 6]
    sums = np.zeros((2, 2))
    for seed in range(6):
        mesh = _mesh(fec, 5, seed)
        X, conn = mesh.nodal_coords, mesh.element_conns["b"] - 1
        asm = fec.SparseMatrixAssembler(fec.VectorFunction(fec.FunctionSpace(mesh), "u"))
        p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3))
        rng = np.random.default_rng(seed)
        U = strain * X @ rng.uniform(-1, 1, (3, 3)) + 0.02 * strain * rng.standard_normal(X.shape)
        R, K, _ = _exact(X.astype(LD), conn, dN, w, p.physics[0].create_properties(), U.astype(LD), U.astype(LD))
        Ud = torch.from_numpy(U.ravel().copy()).cuda()
        for i, switch in enumerate(("1", "0")):
            with environment(FEC_TET4_GENERAL=switch):
                r, k = fec.assemble_residual_and_stiffness(asm, Ud, p)
                sums[i] += [float(np.mean(((got - want) / abs(want).max()) ** 2))
                            for got, want in ((r.cpu().numpy(), R), (k.to_scipy().T.toarray(), K))]
    here, there = np.sqrt(sums / 6)
    print(strain, here, there)
    assert np.all(here <= 1.03 * there)
