"""Order of the stores with which block 0 ends a reduction of the one-launch
solve (csrc/acg_persist.cuh, red_collect).

Block 0 marks the totals of the reduction before pending and publishes the new
ones, both with relaxed stores.  A block that has the new totals may poll the old
ones next, so the reset has to come first and a fence has to lie between; the
memory model allows stale totals otherwise, but a GPU hardly ever shows it.  So
the sequence is checked in the source.
"""
import pathlib
import re

SRC = pathlib.Path(__file__).parents[1] / "laplacians.jl_b200" / "csrc" / "acg_persist.cuh"


def test_totals_are_reset_before_the_fence_of_the_next_publication():
    body = SRC.read_text().split("void red_collect(")[1]
    block0 = body[:body.index("} else {")]
    reset = re.search(r"st_relaxed\(red \+ last \* kRedValues \+ lane, pending_value<double>\(\)\);", block0)
    total = re.search(r"st_relaxed\(red \+ point \* kRedValues \+ lane, smem\[lane\]\);", block0)
    assert reset and total and reset.end() < total.start()
    between = block0[reset.end():total.start()]
    # all lanes reach the fence: another lane's reset is ordered by the warp barrier
    assert re.search(r"__syncwarp\(\);\s*fence_gpu\(\);", between)
