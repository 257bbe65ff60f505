"""The turns that the two tiles of csrc/attention_fmha_pair.cuh take at the exponentials, walked through in every
order of its warps: a barrier says only whether its number of completed phases is odd, so no phase may complete
while a warp has still to look at the one before."""
import itertools
import re

import pytest

from vllm_gcu_b200.csrc import build

WARPS = 2          # of a slot (four in the kernel; two show every order between a fast and a slow one)


def _conditions():
    """When a slot waits for the other's turn, and when it ends its own, as the source says."""
    text = re.sub(r"//[^\n]*", "", (build.CSRC / "attention_fmha_pair.cuh").read_text())
    wait = re.search(r"if \(([^{}]*)\) \{\s*mbar_pass_warp\(&turn\[h \^ 1\]", text).group(1)
    arrive = re.search(r"if \(c == 3 && lane == 0 && ([^;]*)\) mbar_arrive\(&turn\[h\]\)", text).group(1)

    def python(c):
        c = c.replace("&&", " and ").replace("||", " or ")
        m = re.fullmatch(r"\(?(.*?)\?(.*?):(.*?)\)?", c)
        return f"({m[2]}) if ({m[1]}) else ({m[3]})" if m else c
    return python(wait), python(arrive)


def _steps(pieces, wait, arrive):
    """What the warps of both slots do, in order: True waits for the other slot's turn, False ends their own."""
    out = []
    for h in range(2):
        steps, both_before = [], 0
        for tiles in pieces:
            nt_both = min(tiles)
            for j in range(tiles[h]):
                names = dict(h=h, j=j, nt_both=nt_both, both_before=both_before)
                if eval(wait, {}, names):
                    steps.append(True)
                if eval(arrive, {}, names):
                    steps.append(False)
            both_before += nt_both
        out.append(steps)
    return out


def _walk(steps):
    """Every state that the warps can reach; fails where one has to wait for ever or looks too early."""
    waits = [[sum(s[:i]) for i in range(len(s) + 1)] for s in steps]
    ends = [[i - w for i, w in enumerate(v)] for v in waits]
    start = (0,) * (2 * WARPS)
    todo, seen = [start], {start}
    while todo:
        at = todo.pop()
        done = [sum(ends[h][at[h * WARPS + w]] for w in range(WARPS)) // WARPS for h in range(2)]
        moved = False
        for i, p in enumerate(at):
            h = i // WARPS
            if p == len(steps[h]):
                continue
            if steps[h][p]:
                phase = waits[h][p]
                if done[h ^ 1] & 1 == phase & 1:
                    continue                      # the barrier says: not yet
                assert done[h ^ 1] > phase, "a turn is taken before it was given"
            moved = True
            new = at[:i] + (p + 1,) + at[i + 1:]
            if new not in seen:
                seen.add(new)
                todo.append(new)
        assert moved or all(p == len(steps[i // WARPS]) for i, p in enumerate(at)), "a warp waits for ever"


# pieces of work one after the other, with the key tiles of both slots: of heads, which see the same tiles, and of
# two query tiles of a head, of which the second may see one more, or have no rows
@pytest.mark.parametrize("kinds", [[(1, 1), (2, 2), (3, 3)], [(1, 2), (1, 0), (2, 2), (1, 1)]])
def test_every_order_ends(kinds):
    wait, arrive = _conditions()
    for pieces in itertools.product(kinds, repeat=3):
        _walk(_steps(pieces, wait, arrive))


# a slot that does not wait in the first tile of a piece: the walk has to find it
def test_the_walk_finds_a_missing_wait():
    with pytest.raises(AssertionError, match="for ever"):
        _walk(_steps([(2, 2), (1, 1)], "j > 0 if h == 0 else True", "True if h == 0 else j + 1 < nt_both"))
