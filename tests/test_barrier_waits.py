"""Waits by parity in the tensor-core element kernels.  A wait by parity only sees the right
phase if the barrier cannot complete another one before the waiting role has gone on, so a
role may wait for a barrier only if its own later arrival is needed for the next phase.  The
epilogue warps arrive at bar_tfree, which the MMA warp needs before the next tile's bar_mma;
bar_sl completes its next phase without them."""
import re

import pytest

from conftest import ROOT

CSRC = ROOT / "finiteelementcontainers.jl_gb300" / "csrc"


@pytest.mark.parametrize("name", ["fec_hex8_affine_tc.cu", "fec_tet10_tc.cu"])
def test_epilogue_waits_for_the_mmas_alone(name):
    text = (CSRC / name).read_text()
    epilogue = text[text.index("---------------- epilogue:"):text.index("---------------- MMA warp:")]
    assert re.findall(r"wait_or_report\((\w+)", epilogue) == ["bar_mma"]
    assert "mbar_arrive(bar_tfree)" in epilogue
    # the scales in shared memory are read after that wait, and the issuer of the MMAs, which
    # waited for the slices, arrives at bar_mma itself besides the MMAs' commit
    assert epilogue.index("wait_or_report(bar_mma") < epilogue.index("s_tau[")
    mma = text[text.index("---------------- MMA warp:"):]
    assert mma.index("mma_commit(bar_mma)") < mma.index("mbar_arrive(bar_mma)")
    assert "mbar_init(bar_mma, 2)" in text
