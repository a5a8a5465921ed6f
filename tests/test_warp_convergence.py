"""Instructions that a whole warp executes together (.sync.aligned) have a __syncwarp
directly before them in the sources: a warp whose lanes waited each for itself, or left
one lane's branch, need not have come together again.  Nothing else shows a missing one:
the loads would be undefined without an error."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "legitengine_gb300" / "csrc"


def _statements(text):
    """Statements of a source, comments out and strings kept."""
    text = re.sub(r"//[^\n]*", "", text)
    part, depth, quoted, prev = "", 0, False, ""
    for c in text:
        part += c
        if c == '"' and prev != "\\":
            quoted = not quoted
        prev = c
        if quoted:
            continue
        depth += (c == "(") - (c == ")")
        if c in ";{}" and depth <= 0:
            yield part.strip()
            part = ""


@pytest.mark.parametrize("name", sorted(p.name for p in CSRC.glob("*.cu*") if ".sync.aligned" in p.read_text()))
def test_aligned_instructions_follow_a_syncwarp(name):
    before, seen = "", 0
    for statement in _statements((CSRC / name).read_text()):
        if ".sync.aligned" in statement:
            seen += 1
            assert before == "__syncwarp();", f"{statement[:90]!r} follows {before[-60:]!r}"
        before = statement
    assert seen
