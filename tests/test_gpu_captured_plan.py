"""A captured Newton loop has the gather by output entry in its graph, however few assemblies
its warm-up makes: the plan is there before the capture, so eager assemblies after it
allocate nothing, and replay gives the per-node gathers' bits."""
import pytest

from test_gpu_batched import _system
from test_gpu_hex8_general import environment


# cells a side: a plan after four assemblies without it, and after 14
@pytest.mark.gpu
@pytest.mark.parametrize("iterations", [1, 3])
@pytest.mark.parametrize("n", [64, 22])
def test_plan_is_built_before_the_capture(fec, n, iterations):
    import torch
    from fec_gb300 import batching
    asm, p, U, Uu, _ = _system(fec, batching.box_batch([n]).mesh)
    loop = batching.NewtonLoop([(asm, p, Uu)], iterations=iterations).capture()
    loop.replay()
    got, R, nz = loop.unknowns().clone(), fec.residual(asm).clone(), fec.stiffness(asm).nzval.clone()
    with environment(FEC_GATHER_PAIRS="0"):
        eager = batching.NewtonLoop([(asm, p, Uu)], iterations=iterations)
        eager.run_eager()
    assert torch.equal(eager.unknowns(), got)
    assert torch.equal(fec.residual(asm), R) and torch.equal(fec.stiffness(asm).nzval, nz)
    fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(20):
        fec.assemble_residual_and_stiffness(asm, Uu, p)
    torch.cuda.synchronize()
    lists = ((3 * n + 1) ** 3 + (n + 1) ** 3) // 2 * 20 + n ** 3 * 36 * 4
    assert free - torch.cuda.mem_get_info()[0] < lists // 2


def test_null_context_is_refused(fec):
    from fec_gb300 import _lib
    assert _lib.load().fec_set_gather_plan(None, 1) == _lib.FEC_ERR_ARG
