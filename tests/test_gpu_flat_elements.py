"""FP64 Neo-Hookean hex8 and tet10 elements of aspect ratios up to 10,000, distorted and
sheared, against the same sums in extended precision: residual, tangent and matrix-free
action of the kernels that work in reference coordinates are no further off than the
per-element kernels.

Tolerance: both are roundings of one set of sums, so they share its condition; a factor of
three between two such errors, plus the 2^-48 of a double-float entry a few times over."""
import numpy as np
import pytest

import test_gpu_hex8_general as hex8
import test_gpu_tet10_general as tet10
from test_gpu_hex8_general import environment

pytestmark = pytest.mark.gpu
LD = np.longdouble
FLOOR = 4 * 2.0 ** -48


def _exact(X, conn, dN, w, props, U, V):
    """Residual, tangent and K v of the mesh, dense, in extended precision."""
    K_, G_ = (LD(p) for p in props[:2])
    n = X.size
    R, K, dof = np.zeros(n, LD), np.zeros((n, n), LD), (3 * conn[:, :, None] + np.arange(3)).reshape(len(conn), -1)
    I = np.eye(3, dtype=LD)
    for d, wq in zip(dN, w):
        G = np.einsum("eai,aj->eij", X[conn], d)
        det = lambda A: np.einsum("ei,ei->e", A[:, 0], np.cross(A[:, 1], A[:, 2]))  # noqa: E731
        cof = lambda A: np.stack([np.cross(A[:, 1], A[:, 2]), np.cross(A[:, 2], A[:, 0]), np.cross(A[:, 0], A[:, 1])], 1)  # noqa: E731
        g = np.einsum("aj,eij->eai", d, cof(G) / det(G)[:, None, None])
        jxw = (det(G) * wq)[:, None, None]
        F = I + np.einsum("eai,eaj->eij", U[conn], g)
        J = det(F)[:, None, None]
        y = np.cbrt(J)
        y = y - (y * y * y - J) / (3 * y * y)
        H, c2 = cof(F) / J, G_ / (y * y)
        I13 = (F * F).sum((1, 2), keepdims=True) / 3
        c1 = K_ / 2 * (J * J - J - 1)
        P = c1 * H + c2 * (F - I13 * H)
        a1, a2 = K_ / 2 * (2 * J - 1) * J + LD(2) / 3 * c2 * I13, I13 * c2 - c1
        e4 = lambda s: s[:, :, :, None, None]  # noqa: E731
        o = lambda A, B: np.einsum("eij,ekl->eijkl", A, B)  # noqa: E731
        A = (e4(a1) * o(H, H) + e4(a2) * np.einsum("eil,ekj->eijkl", H, H) - LD(2) / 3 * e4(c2) * (o(F, H) + o(H, F))
             + e4(c2) * np.einsum("ik,jl->ijkl", I, I)[None])
        np.add.at(R, dof, np.einsum("eaj,eij->eai", g, P * jxw).reshape(dof.shape))
        Ke = np.einsum("eaj,eijkl,ebl->eaibk", g, A * e4(jxw), g).reshape(len(conn), dof.shape[1], -1)
        np.add.at(K, (dof[:, :, None], dof[:, None, :]), Ke)
    return R, K, K @ V.ravel()


def _hex_rule():
    t = 1 / np.sqrt(LD(3))
    at = np.array([[i & 1, i >> 1 & 1, i >> 2] for i in range(8)]) * 2 - 1
    node = at[[0, 1, 3, 2, 4, 5, 7, 6]]
    dN = np.zeros((8, 8, 3), LD)
    for q in range(8):
        f = (1 + node * (at[q] * t)) / 2
        for j in range(3):
            dN[q, :, j] = LD(1) / 2 * node[:, j] * f[:, (j + 1) % 3] * f[:, (j + 2) % 3]
    return dN, np.ones(8, LD)


def _tet_rule():
    b = (5 - np.sqrt(LD(5))) / 20
    gl = np.concatenate([-np.ones((1, 3), LD), np.eye(3, dtype=LD)])
    dN = np.zeros((4, 10, 3), LD)
    for q in range(4):
        lam = np.full(4, b)
        lam[q] = 1 - 3 * b
        dN[q, :4] = (4 * lam - 1)[:, None] * gl
        for k, (m, n) in enumerate(tet10.EDGES):
            dN[q, 4 + k] = 4 * (lam[m] * gl[n] + lam[n] * gl[m])
    return dN, np.full(4, LD(1) / 24)


@pytest.mark.parametrize("strain", [1e-3, 0.05])
@pytest.mark.parametrize("aspect", [1, 100, 1000, 10000])
@pytest.mark.parametrize("kind", ["hex8", "tet10"])
def test_no_further_off_than_the_per_element_kernels(fec, kind, aspect, strain):
    import torch
    flat = (1.0, 1.0, 1.0 / aspect)
    if kind == "hex8":
        mesh, (dN, w), switch = hex8._mesh(fec, (3, 4, 3), 4, flat), _hex_rule(), "FEC_HEX8_GENERAL"
    else:
        mesh, (dN, w), switch = tet10._mesh(fec, (2, 2, 2), 48, stretch=flat, bend=0.02), _tet_rule(), "FEC_TET10_GENERAL"
    X, conn = mesh.nodal_coords, mesh.element_conns["b"] - 1
    u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
    asm = fec.SparseMatrixAssembler(u)
    p = fec.create_parameters(mesh, asm, fec.NeoHookean.from_youngs(1.0, 0.3))
    rng = np.random.default_rng(aspect)
    U = strain * X @ np.array([[1.0, 0.3, 0.4], [-0.2, -0.6, 0.5], [0.8, 0.7, -0.5]])
    U += 0.1 * strain / 3 / aspect * rng.standard_normal(X.shape)
    V = rng.standard_normal(X.shape)
    R, K, A = _exact(X.astype(LD), conn, dN, w, p.physics[0].create_properties(), U.astype(LD), V.astype(LD))
    Ud, Vd = torch.from_numpy(U.ravel().copy()).cuda(), torch.from_numpy(V.ravel().copy()).cuda()

    def errors():
        r, k = fec.assemble_residual_and_stiffness(asm, Ud, p)
        r, k = r.cpu().numpy().copy(), k.to_scipy().T.toarray()
        fec.assemble_vector(asm, fec.residual, Ud, p)
        assert np.array_equal(fec.residual(asm).cpu().numpy(), r)
        a = fec.assemble_matrix_free_action(asm, fec.stiffness_action, Ud, Vd, p).cpu().numpy()
        return {n: float(abs(got - want).max() / abs(want).max()) for n, got, want in (("R", r, R), ("K", k, K), ("action", a, A))}

    here = errors()
    with environment(**{switch: "0"}):
        there = errors()
    print(kind, aspect, strain, here, there)
    for n in here:
        assert here[n] <= 3 * there[n] + FLOOR, (n, here, there)
