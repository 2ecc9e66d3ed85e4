"""The order between the sweep ring's two kinds of access (awfl_sweep.cuh), read from the source:
a race between proxies shows in no result that a test could compare.

A persistent CTA (the ensembles) sweeps tile after tile on one shared-memory ring. The first
TMA boxes of a tile are issued at its start, so every thread's generic-proxy accesses to the
ring in the tile before -- cp.async rows, halo values, reads -- must have passed a proxy fence
and then a barrier before that: at the end of the tile."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "awflcloud_b200", "csrc")


def _body(path, head):
    """The braces' contents of the function whose text begins with `head`, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(SRC, path)).read())
    at = text.index("{", text.index(")", text.index(head)))
    depth, i = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return text[at:i]


def test_tile_ends_with_a_proxy_fence_and_a_barrier():
    body = _body("awfl_sweep.cuh", "void sweep_tile(")
    issue = body.index("if (cur_tma) issue_tma(HS);")
    uses = [m.start() for m in re.finditer(r"\b(ringAt|stage|finish|finish_first)\s*\(", body)]
    tail = body[max(uses):]
    # after the last generic access, for every thread of the TMA form: fence, then barrier
    assert re.search(r"if constexpr \(TMA\) \{\s*fence_proxy_async\(\);\s*__syncthreads\(\);", tail), tail
    # and what the early issue relies on within the tile: the prologue's own fence before its barrier
    assert re.search(r"if constexpr \(TMA\) \{\s*fence_proxy_async\(\);\s*__syncthreads\(\);", body[issue:max(uses)])


def test_first_boxes_fill_no_slot_of_the_prologue():
    """Position p of a line lies in slot (p - HS) mod 4C; the prologue writes positions -HS..HS-1,
    the first chunk's boxes fill HS..HS+C-1."""
    body = _body("awfl_sweep.cuh", "void sweep_tile(")
    assert "const int s = (p - HS) & (R - 1);" in body
    assert re.search(r"constexpr int R = ASYNC \? 4 \* C", body)
    for HS in (2, 4):
        for C in (4, 8, 16, 32):
            if C < 2 * HS:
                continue
            pro = {(p - HS) % (4 * C) for p in range(-HS, HS)}
            box = {(p - HS) % (4 * C) for p in range(HS, HS + C)}
            assert not pro & box
