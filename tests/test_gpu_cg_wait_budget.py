"""The barriers of the one-launch solve wait for the budget that is set: one clock either is
enough or ends the solve with an error status, and the next solve is right."""
import numpy as np
import pytest

from test_gpu_cg_kernels import _solve, _system

pytestmark = pytest.mark.gpu


def test_a_barrier_that_gives_up_is_an_error_and_the_next_solve_is_right(fec):
    import torch
    asm, K = _system(fec, "quad4", (60,))     # 3,481 unknowns: 14 CTAs
    n = asm.dof.unknown_dofs.size
    b = torch.from_numpy(np.random.default_rng(1).standard_normal(n)).cuda()
    x = torch.zeros_like(b)
    want = _solve(asm, K, b, x, 2000, 1e-12, True)
    assert want[1] <= 1e-12
    lib, errors = fec.load_library(), 0
    for _ in range(5):
        assert lib.fec_set_wait_budget(1) == 0
        try:
            y = torch.zeros_like(b)
            assert _solve(asm, K, b, y, 2000, 1e-12, True) == want and torch.equal(y, x)
        except fec.FECError as e:
            errors += 1
            assert "timed out" in str(e) or "timeout" in str(e)
        finally:
            lib.fec_set_wait_budget(0)
        y = torch.zeros_like(b)
        assert _solve(asm, K, b, y, 2000, 1e-12, True) == want and torch.equal(y, x)
    # (200 iterations of three barriers over 14 CTAs: none arrives within a clock of the last)
    assert errors == 5
