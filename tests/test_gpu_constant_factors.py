"""FP64 hex8 blocks whose mapping is a table of the block (translated elements, and the
reference element of the kernels for any shape): rounding of the table is a common factor of all
entries, which no sum averages out.  Errors of the matrix-free action,
against the same sums in extended precision, are no larger in the mean than the per-element
kernels', which form the mapping point by point: root mean squares over eight meshes of 36
elements (some 240 values each, so equal precision shows within a few per cent)."""
import numpy as np
import pytest

from test_gpu_flat_elements import LD, _exact, _hex_rule
from test_gpu_hex8_general import _mesh, environment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strain", [1e-3, 0.05])
@pytest.mark.parametrize("kind", ["bent", "box", "skew"])
def test_action_error_is_no_larger_than_the_per_element_kernels(fec, kind, strain):
    import torch
    dN, w = _hex_rule()
    sums = {"here": 0.0, "per element": 0.0}
    for seed in range(8):
        mesh = _mesh(fec, (3, 4, 3), seed)
        conn = mesh.element_conns["b"]
        X = mesh.nodal_coords
        if kind != "bent":
            z, y, x = np.meshgrid(np.arange(4), np.arange(5), np.arange(4), indexing="ij")
            X = np.stack([x.ravel(), y.ravel(), z.ravel()], 1) * np.array([0.375, 0.25, 0.3125])
            if kind == "skew":
                X = X @ np.array([[1.0, 0.25, 0.0], [0.125, 0.875, 0.25], [0.0, -0.25, 1.125]])
            mesh = fec.UnstructuredMesh(X, {"b": ("HEX8", conn)})
        asm = fec.SparseMatrixAssembler(fec.VectorFunction(fec.FunctionSpace(mesh), "u"))
        p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3))
        rng = np.random.default_rng(seed)
        U = strain * X @ rng.uniform(-1, 1, (3, 3)) + 0.01 * strain * rng.standard_normal(X.shape)
        V = rng.standard_normal(X.shape)
        _, _, A = _exact(X.astype(LD), conn - 1, dN, w, p.physics[0].create_properties(), U.astype(LD), V.astype(LD))
        Ud, Vd = torch.from_numpy(U.ravel().copy()).cuda(), torch.from_numpy(V.ravel().copy()).cuda()

        def error():
            a = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Ud, Vd, p).cpu().numpy()
            return float(np.mean(((a - A) / abs(A).max()) ** 2))

        sums["here"] += error()
        with environment(FEC_HEX8_GENERAL="0", FEC_HEX8_AFFINE="0"):
            sums["per element"] += error()
    print(kind, strain, {k: (v / 8) ** 0.5 for k, v in sums.items()})
    assert sums["here"] ** 0.5 <= 1.05 * sums["per element"] ** 0.5
