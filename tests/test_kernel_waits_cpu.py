"""A wait that runs out leaves the lanes of a warp together: outside of blocks that one elected lane runs,
the kernels wait through mbar_wait_warp, whose answer is the same in all lanes.  Behind such a wait come
tensor-memory copies and barriers that want whole warps, and nothing else keeps lanes together whose
look at the barrier ended at different times."""
import re

import pytest

from vllm_gcu_b200.csrc import build


def _waits(text):
    """(line, headers of the enclosing blocks) of every mbar_wait call."""
    text = re.sub(r"//[^\n]*", "", text)
    blocks, start, found = [], 0, []
    for i, c in enumerate(text):
        if c == "{":
            blocks.append(text[start:i])
            start = i + 1
        elif c == "}":
            blocks.pop()
            start = i + 1
        elif c == ";":
            start = i + 1
        elif c == "(" and re.search(r"\bmbar_wait$", text[max(0, i - 12):i]):
            found.append((text.count("\n", 0, i) + 1, list(blocks)))
    return found


@pytest.mark.parametrize("source", ["attention_fmha_pair.cuh", "attention_mla.cu", "gemm_pair_rows.cu",
                                    "gemm_stream.cu", "gemm_wna16_stream.cu"])
def test_whole_warps_wait_as_one(source):
    text = (build.CSRC / source).read_text()
    waits = _waits(text)
    assert waits and "mbar_wait_warp(" in text
    alone = [line for line, blocks in waits if not any("elect_one()" in b for b in blocks)]
    assert not alone, f"{source}: lanes that wait one by one in lines {alone}"


def test_one_answer_for_a_warp():
    text = (build.CSRC / "common.cuh").read_text()
    body = text[text.index("bool mbar_wait_warp("):]
    assert re.search(r"return __all_sync\(0xffffffffu,\s*mbar_wait\(", body[:body.index("\n}")])
