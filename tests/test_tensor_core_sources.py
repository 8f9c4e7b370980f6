"""Orderings of the tensor-core kernels that a run on a healthy GPU cannot show
missing, read from their sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).parent.parent / "pyaxisymflow_gb300" / "csrc"


def role(source, name):
    """The statements of one warp's branch (warp == 0: copies, warp == 1: MMAs)."""
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    start = text.index(f"if (warp == {name}) {{\n    if (elect_one())")
    return text[start:text.index("__syncwarp();", start)]


@pytest.mark.parametrize("source", ["sliced_gemm.cu", "tc_gemm.cu"])
def test_a_failed_block_waits_for_its_mmas(source):
    """After a failure the error word is set and mbar_wait gives up after a few
    polls; the wait for the block's MMAs must not."""
    mma = role(source, 1)
    after = mma[mma.index("umma_commit(quiet)"):]
    assert "mbar_wait_drain(quiet" in after
    assert not re.search(r"\bmbar_wait\(quiet", after)


@pytest.mark.parametrize("source", ["sliced_gemm.cu", "tc_gemm.cu"])
@pytest.mark.parametrize("warp", [0, 1])
def test_time_limits_start_after_the_predecessor(source, warp):
    """A kernel of a chain may start while its predecessor runs; no wait with a
    time limit starts before it has waited for that one."""
    text = role(source, warp)
    assert text.index("pdl_wait()") < re.search(r"\bmbar_wait\(", text).start()
