"""The warps of traverse_queue share the length of their triangle list.  Every
lane has to see the same length, since all of them or none enter the tests
that it starts: a __syncwarp() stands between any two accesses of it that do
not commute (a ballot makes the lanes meet, but orders no memory).

Read from the source: in the loop's order, around its end included, with the
branch that skips the tests taken and not taken.
"""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parents[1] / "optixrender_b200" / "csrc" / "rt_traverse.cuh"


def _block(text, at):
    """The text from the brace at or after `at` to the one that closes it."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced braces")


def _accesses(body):
    kinds = {"atomicAdd(&w.count": "add", "w.count = 0": "write", "__syncwarp()": "sync", "w.count": "read",
             "test_triangles<": "sync"}  # the tests meet in __syncwarp() themselves
    return [kinds[m.group(0)] for m in re.finditer("|".join(re.escape(k) for k in kinds), body)]


def test_every_lane_sees_the_same_list_length():
    text = re.sub(r"//[^\n]*", "", SOURCE.read_text())
    function = _block(text, text.index("RT_D void traverse_queue("))
    loop = _block(function, function.index("while (true)"))
    tests = _block(loop, loop.index("if (n > 0 &&"))
    for body in (loop, loop.replace(tests, "{}")):
        order = _accesses(body)
        assert {"add", "read", "sync"} <= set(order)
        order += order  # the next round
        last = None
        for kind in order:
            if kind == "sync":
                last = None
            elif last is not None and {last, kind} != {"add"} and {last, kind} != {"read"}:
                raise AssertionError(f"{last} and {kind} of the list's length without a __syncwarp() between them")
            else:
                last = kind
