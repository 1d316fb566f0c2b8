"""The rings of the 32-bit product on the tensor cores (csrc/gemm_f32_tcgen05.cu), read from its source and walked on the
CPU: copies land in any order, teams of warps cut every n-th block, and a wait on an mbarrier goes by the parity of its
phase alone.  No team may cut a block that has not landed."""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "flyweight_b200" / "csrc" / "gemm_f32_tcgen05.cu"


def shape_of(text, tile):
    """(slots for copies, stages of cut blocks, teams) of a tile, from ``name = NT > a ? x : NT > b ? y : z``."""
    found = []
    for name in ("RAW_STAGES", "STAGES", "TEAMS"):
        chain = re.search(rf"\b{name} = (NT >[^;,]*)", text).group(1).split(":")
        for part in chain:
            cond = re.match(r"\s*NT > (\d+) \? (\d+)", part)
            if cond is None or tile > int(cond.group(1)):
                found.append(int(cond.group(2) if cond else part))
                break
    return tuple(found)


def waits_of(text):
    """The barriers that a cutting warp waits for ahead of a block, in order."""
    cutter = text[text.index("if (warp < CUTTERS)"):text.index("else if (warp == LOAD_WARP)")]
    return re.findall(r"mbar_wait\(&(\w+)\[", re.sub(r"//[^\n]*", "", cutter))


def cut_too_early(slots, stages, teams, waits, blocks=9):
    """Every order of events of `blocks` blocks: the first block found that is cut before it has landed, or None."""
    def passes(completed, parity):                      # the phase of that parity is over, as far as an mbarrier can tell
        return completed % 2 != parity

    # (copies asked for, landed, a team's next block and how many of its waits are behind it, cut, multiplied)
    start = (0, frozenset(), tuple((team, 0) for team in range(teams)), frozenset(), 0)
    seen, todo = {start}, [start]
    while todo:
        asked, landed, at, cut, done = todo.pop()
        follow = []
        # the loading lane: a slot is free when its tenant has been cut (it sees every block, so no phase passes it by)
        if asked < blocks and (asked < slots or asked - slots in cut):
            follow.append((asked + 1, landed, at, cut, done))
        follow += [(asked, landed | {b}, at, cut, done) for b in range(asked) if b not in landed]
        if done < blocks and done in cut:               # the multiplying warp, block after block
            follow.append((asked, landed, at, cut, done + 1))
        for team, (block, behind) in enumerate(at):
            if block >= blocks:
                continue
            if behind < len(waits):
                if waits[behind] == "raw_full":
                    over = sum(b % slots == block % slots for b in landed)
                    go = passes(over, block // slots % 2)
                else:
                    over = len(range(block % stages, done, stages))
                    go = block < stages or passes(over, (block // stages - 1) % 2)
                if go:
                    follow.append((asked, landed, at[:team] + ((block, behind + 1),) + at[team + 1:], cut, done))
                continue
            if block not in landed or (block >= stages and done <= block - stages):
                return block
            follow.append((asked, landed, at[:team] + ((block + teams, 0),) + at[team + 1:], cut | {block}, done))
        for state in follow:
            if state not in seen:
                seen.add(state)
                todo.append(state)
    return None


@pytest.mark.parametrize("tile", [16, 64, 112, 208])
def test_no_block_is_cut_before_it_has_landed(tile):
    text = SOURCE.read_text()
    waits = waits_of(text)
    assert sorted(waits) == ["empty_bar", "raw_full"]
    assert cut_too_early(*shape_of(text, tile), waits) is None


def test_waits_in_the_other_order_are_found():
    assert shape_of(SOURCE.read_text(), 208) == (3, 2, 2)
    assert cut_too_early(3, 2, 2, ["raw_full", "empty_bar"]) is not None
    assert cut_too_early(5, 3, 3, ["raw_full", "empty_bar"]) is not None
    assert cut_too_early(6, 4, 3, ["raw_full", "empty_bar"]) is None
