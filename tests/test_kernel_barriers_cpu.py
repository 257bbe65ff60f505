"""Barriers whose form wants all lanes of a warp at once stand behind a __syncwarp(): lanes that took different
ways in front of them (a loop over columns that does not divide evenly, a store of a few lanes) are not together
again by themselves."""
import re

from vllm_gcu_b200.csrc import build


def _sources():
    return sorted([*build.CSRC.glob("*.cu"), *build.CSRC.glob("*.cuh")])


def test_cluster_barriers_and_barriers_of_two_warps():
    found = 0
    for path in _sources():
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r'asm volatile\("(barrier\.cluster\.\w+\.\w+\.aligned|bar\.sync %\d, 64);', text):
            before = text[:m.start()].rstrip()
            assert before.endswith("__syncwarp();"), (path.name, text.count("\n", 0, m.start()) + 1)
            found += 1
    assert found >= 3
