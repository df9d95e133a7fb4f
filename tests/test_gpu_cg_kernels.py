"""The conjugate-gradient kernels at the sizes where their work split ends: fewer
rows than a warp or a CTA takes, partial last groups, rows longer than one
staged round, iteration limits that are not a multiple of the test interval, and
a zero right-hand side."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse.linalg as spl

pytestmark = pytest.mark.gpu


def _system(fec, kind, cells):
    import torch
    if kind == "hex27":   # rows of up to 375 entries
        from fec_gb300.meshes import box_hex27
        mesh = box_hex27(tuple(n + 1 for n in cells))
        n = [2 * c + 1 for c in cells]
        ids = np.arange(1, n[0] * n[1] * n[2] + 1).reshape(n[2], n[1], n[0])
        mesh.nodeset_nodes["bottom"] = ids[0].ravel()
        u = fec.VectorFunction(fec.FunctionSpace(mesh), "u")
        phys, faces, names = fec.J2Plasticity(200.0, 0.3, 0.25, 2.0), ["bottom"], u.names
    else:
        mesh = fec.StructuredMesh("quad", (0.0, 0.0), (1.0, 1.0), (cells[0] + 1, cells[0] + 1))
        u = fec.ScalarFunction(fec.FunctionSpace(mesh), "u")
        phys, faces, names = fec.Poisson(1.0), ["bottom", "top", "left", "right"], u.names
    asm = fec.SparseMatrixAssembler(u)
    bcs = [fec.DirichletBC(v, lambda X, t: 0.0, nodeset_name=f) for f in faces for v in names]
    p = fec.create_parameters(mesh, asm, phys, dirichlet_bcs=bcs)
    _, K = fec.assemble_residual_and_stiffness(asm, torch.zeros(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda(),
                                               p)
    return asm, K


def _solve(asm, K, b, x, max_iter, rtol, jacobi):
    import torch
    from fec_gb300 import _lib
    it, rr = C.c_int(-1), C.c_double(-1.0)
    asm._call("fec_cg_solve", _lib.ptr(K.nzval), _lib.ptr(b), _lib.ptr(x), max_iter, rtol, int(jacobi), C.byref(it),
              C.byref(rr), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return it.value, rr.value


# 1 unknown; 9; 36 (a warp and four rows); 256; 289 (a CTA's rows and one more); 40,000; rows of 375 entries
@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("kind, cells", [("quad4", (2,)), ("quad4", (4,)), ("quad4", (7,)), ("quad4", (17,)),
                                         ("quad4", (18,)), ("quad4", (201,)), ("hex27", (3, 3, 2))])
def test_solution_matches_direct_solve(fec, kind, cells, jacobi):
    import torch
    asm, K = _system(fec, kind, cells)
    n = asm.dof.unknown_dofs.size
    rng = np.random.default_rng(n)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    x = torch.from_numpy(x0.copy()).cuda()
    it, rr = _solve(asm, K, torch.from_numpy(b).cuda(), x, 20000, 1e-12, jacobi)
    ref = spl.spsolve(K.to_scipy().tocsc(), b)
    # ||b - K x|| <= 1e-12 ||b||: the solution to that times the condition number (below 1e4 here)
    assert it % 10 == 0 and 0 < it < 20000 and rr <= 1e-12
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-8 * np.linalg.norm(ref)


@pytest.mark.parametrize("max_iter", [0, 1, 7, 10, 13])
def test_iteration_limit(fec, max_iter):
    import torch
    asm, K = _system(fec, "quad4", (40,))
    n = asm.dof.unknown_dofs.size
    rng = np.random.default_rng(1)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    x = torch.from_numpy(x0.copy()).cuda()
    it, rr = _solve(asm, K, torch.from_numpy(b).cuda(), x, max_iter, 1e-14, False)
    A = K.to_scipy()
    xr = x0.copy()
    r = b - A @ xr
    d = r.copy()
    for _ in range(max_iter):   # the same iterations in numpy
        y = A @ d
        alpha = (r @ r) / (d @ y)
        xr, new = xr + alpha * d, r - alpha * y
        d, r = new + (new @ new) / (r @ r) * d, new
    assert it == max_iter
    assert np.linalg.norm(x.cpu().numpy() - xr) <= 1e-12 * np.linalg.norm(xr)
    assert abs(rr - (np.linalg.norm(r) / np.linalg.norm(b) if max_iter else 0.0)) <= 1e-9


def test_zero_right_hand_side(fec):
    import torch
    asm, K = _system(fec, "quad4", (9,))
    x = torch.ones(asm.dof.unknown_dofs.size, dtype=torch.float64).cuda()
    it, rr = _solve(asm, K, torch.zeros_like(x), x, 100, 1e-12, True)
    assert (it, rr) == (0, 0.0) and float(x.abs().max()) == 0.0
