"""The chunk products' marks of values that are not finite, on the host: the place of a unit's mark is that of the unit before
the last, so that unit's marks must have been read and cleared first.  The order in which the kernel's warps wait for one
another is laid out as a graph of events; what is no ancestor of a mark may come behind it."""
import os

import pytest

import picolm_b200

SOURCE = os.path.join(os.path.dirname(picolm_b200.__file__), "csrc", "scan_chunk.cu")


def _marks_behind_the_wait():
    """Whether the kernel marks behind its wait for the MMAs that read a buffer last."""
    with open(SOURCE) as f:
        text = f.read()
    text = text[text.index("chunk_product_kernel("):]
    return text.index("(mma_done(group)") < text.index("atomicMin(&reached_from")


def _before(event, behind, ring, steps):
    """All events that come before `event` whatever the warps' speeds."""
    def needs(e):
        kind, s = e
        if kind == "loaded":
            return [("loaded", s - 1), ("split", s - ring)]
        if kind == "mark":
            return [("loaded", s), ("split", s - 2)] + ([("mma", s - 2)] if behind else [])
        if kind == "split":
            return [("mark", s), ("mma", s - 2)]
        if kind == "mma":
            return [("split", s), ("read", s - 2), ("mma", s - 2)]
        if kind == "read":
            return [("mma", s), ("read", s - 1)] + ([("clear", s // steps - 1)] if s % steps == 0 else [])
        return [("read", s * steps + steps - 1)]                 # clear: behind a unit's last sums
    seen, todo = set(), [event]
    while todo:
        for e in needs(todo.pop()):
            if e[1] >= 0 and e not in seen:
                seen.add(e)
                todo.append(e)
    return seen


@pytest.mark.parametrize("steps", [4, 6])                        # keys of up to 64, of up to 128
def test_a_mark_finds_its_place_cleared(steps):
    behind = _marks_behind_the_wait()
    for unit in range(2, 7):
        for s in range(unit * steps, (unit + 1) * steps):
            assert ("clear", unit - 2) in _before(("mark", s), behind, 4, steps), (unit, s)


def test_marks_before_the_wait_would_not():
    assert ("clear", 0) not in _before(("mark", 8), False, 4, 4)
    assert ("clear", 0) in _before(("mark", 12), False, 4, 6)
