"""Conjugate gradients where the residual becomes exactly zero between two stopping tests (one
unknown, equal eigenvalues, a start that already solves the system): x stays finite and solves
it, in the one-launch solve and with three kernels an iteration."""
import numpy as np
import pytest

from test_gpu_cg_kernels import _solve, _system
from test_gpu_hex8_general import environment

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rtol", [1e-10, 0.0])
@pytest.mark.parametrize("max_iter", [3, 10, 35])
@pytest.mark.parametrize("jacobi", [False, True])
@pytest.mark.parametrize("coop", ["1", "0"])
@pytest.mark.parametrize("kind", ["one unknown", "equal eigenvalues", "already exact"])
def test_x_is_finite_and_solves_the_system(fec, kind, coop, jacobi, max_iter, rtol):
    import torch
    asm, K = _system(fec, "quad4", (2 if kind == "one unknown" else 18,))
    n = asm.dof.unknown_dofs.size
    assert n == (1 if kind == "one unknown" else 289)
    if kind != "one unknown":   # 2 I: every product and quotient below is exact
        A = K.to_scipy().tocoo()
        K.nzval.copy_(torch.from_numpy(np.where(A.row == A.col, 2.0, 0.0)))
    for seed in range(20 if kind == "one unknown" else 2):
        rng = np.random.default_rng(seed)
        b = rng.standard_normal(n)
        ref = b / K.to_scipy().diagonal()
        x = torch.from_numpy(ref.copy() if kind == "already exact" else np.zeros(n)).cuda()
        with environment(FEC_CG_COOP=coop):
            it, rr = _solve(asm, K, torch.from_numpy(b).cuda(), x, max_iter, rtol, jacobi)
        assert it == (min(max_iter, 10) if rtol else max_iter)
        # one unknown: rounding of two products and a quotient; else exact
        assert rr <= (4e-16 if kind == "one unknown" else 0.0)
        assert np.abs(x.cpu().numpy() - ref).max() <= (1e-15 if kind == "one unknown" else 0.0) * np.abs(ref).max()
