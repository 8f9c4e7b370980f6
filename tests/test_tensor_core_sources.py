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


def test_standalone_plan_depends_on_the_grid_alone():
    """The plan and the run of a transform form its layout each; neither asks the
    device that happens to be current."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "sliced_gemm.cu").read_text())
    start = text.index("TransformLayout transform_layout(")
    assert "sm_count" not in text[start:text.index("\n}\n", start)]


@pytest.mark.parametrize("source", ["sliced_gemm.cu", "tc_gemm.cu"])
def test_a_block_waits_for_the_releases_of_its_last_stages(source):
    """Commits arrive on the stages' barriers by themselves; the copying warp waits
    for the last ones before the block ends."""
    text = role(source, 0)
    tail = text[text.index("progress[0] = g"):]
    assert re.search(r"g \+ q >= NSTAGE\) ok = mbar_wait\(empty0 \+ 8 \* s, lap", tail)
