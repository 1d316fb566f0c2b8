"""A bounded wait that gives up may answer the lanes of a warp differently (one saw the barrier's phase in its last poll,
the next did not).  Lanes that then go different ways meet again at no warp-wide instruction, and the wait that was
bounded has become one that is not.  Read from the sources: nothing here makes a wait run out."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "flyweight_b200" / "csrc"
WAIT = re.compile(r"\bmbar_wait(_cluster)?\(")
ONE_THREAD = ("lane == 0", "threadIdx.x == 0")


def unvoted_waits(text):
    """The waits whose answer code that a whole warp runs goes by, without a vote in the same statement or, on the
    variable that took the answer, in one of the next two."""
    text = re.sub(r"//[^\n]*", "", text)
    headers, start, found = [], 0, []
    for at, ch in enumerate(text):
        if ch not in ";{}":
            continue
        statement = text[start:at]
        if WAIT.search(statement) and not any(one in header for header in headers for one in ONE_THREAD):
            ignored = re.match(r"\s*(tc5::)?mbar_wait", statement)              # the code goes one way whatever it says
            taken = re.search(r"(\w+) = [^;]*?mbar_wait", statement)
            voted = "__all_sync" in statement or taken and any(
                re.search(rf"__all_sync\([^;]*\b{taken.group(1)}\b", later) for later in text[at + 1:].split(";", 2)[:2])
            if not (ignored or voted):
                found.append(" ".join(statement.split()))
        if ch == "{":
            headers.append(statement)
        elif ch == "}" and headers:
            headers.pop()
        start = at + 1
    return found


@pytest.mark.parametrize("name", sorted(path.name for path in CSRC.glob("*.cu") if WAIT.search(path.read_text())))
def test_a_warp_goes_one_way_behind_a_bounded_wait(name):
    assert unvoted_waits((CSRC / name).read_text()) == []


def test_a_wait_without_a_vote_is_found():
    lone = "void k() { if (lane == 0) { ok = mbar_wait(&b, 0); if (!ok) return; } }"
    bare = "void k() { for (;;) { ok = mbar_wait(&b, 0); if (!ok) break; } }"
    vote = "void k() { for (;;) { ok = mbar_wait(&b, 0); ok = ok && !*flag; ok = __all_sync(~0u, ok); if (!ok) break; } }"
    assert unvoted_waits(lone) == [] and unvoted_waits(vote) == []
    assert unvoted_waits(bare) == ["ok = mbar_wait(&b, 0)"]
