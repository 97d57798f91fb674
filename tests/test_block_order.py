"""Ordering of the controller's fields in the block solver, checked on its source: what warp 0 writes for
the next attempt must not be read by a warp that has nothing left to meet it at."""
import os
import re

from conftest import ROOT

SOURCE = open(os.path.join(ROOT, "disco-eb_b200", "csrc", "solve_block.cuh")).read()


def _code(text):
    return re.sub(r"//[^\n]*", "", text)


def _body(head):
    """The braces' content of the function or block that starts at head."""
    start = SOURCE.index("{", SOURCE.index(head))
    depth = 0
    for i in range(start, len(SOURCE)):
        depth += {"{": 1, "}": -1}.get(SOURCE[i], 0)
        if depth == 0:
            return _code(SOURCE[start + 1:i])
    raise AssertionError(head)


def _controller():
    """Warp 0 between the end of one attempt and the barrier that starts the next."""
    solve = _body("solve_mode_block(")
    start = solve.rindex("if (warp == 0) {", 0, solve.index("R.steps++"))
    return solve[start:solve.index("bar_sync(0, c_solve);", start)]


def _controller_fields():
    fields = set(re.findall(r"S\.c\.(\w+) = ", _controller()))
    assert {"t", "h", "tnext", "regime", "go", "accepted", "e2", "e3"} <= fields
    return fields


def test_helper_warps_read_the_controllers_fields_before_their_first_barrier():
    """After their last stage's barriers neither the scale nor the prep warp meets warp 0 again before it
    writes these fields for the next attempt."""
    body = _body("helper_step(")
    split, other = body.index("if (warp_a) {"), body.rindex("\n    } else {")
    assert not re.search(r"\bbar_(sync|arrive)\(", body[:split])
    for branch in (body[split:other], body[other:]):
        late = branch[re.search(r"\bbar_(sync|arrive)\(", branch).start():]
        assert not set(re.findall(r"S\.c\.(\w+)", late)) & _controller_fields()
    assert "S.c." not in _body("prep_point(")


def test_controller_writes_its_fields_after_every_lane_has_read_the_old_ones():
    """All lanes of warp 0 read the attempt's outcome and its leader overwrites it: the lanes meet between."""
    text = _controller()
    write = min(m.start() for m in re.finditer(r"S\.c\.(\w+) = ", text))
    reads = [m.start() for m in re.finditer(r"S\.c\.(\w+)(?! = )\b", text) if m.start() < write]
    assert reads
    assert "tm.sync();" in text[max(reads):write]
    leader = text.rindex("if (tm.leader()) {", 0, write)
    assert text[:leader].rstrip().endswith("tm.sync();")
