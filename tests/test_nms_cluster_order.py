"""The runs of equal scores that the first block of an NMS cluster hands to the others
(geye_gb300/csrc/nms_batch.cu, settle_members): every block copies them out of the first block's shared
memory and decides by its copy how the sort goes on; where all boxes are to be sorted (split_boxes)
each block then writes its own again.  The steps are read from the source, in order, and run under
random schedules: every copy must be of the runs, complete, before the first block overwrites them."""
import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geye_gb300", "csrc", "nms_batch.cu")
BLOCKS = 16


def _body(src, name):
    """The text of a device function's body."""
    start = re.search(r"\b" + name + r"\([^;{]*\)\s*\{", src).end()
    depth = 1
    for k in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        if depth == 0:
            return src[start:k]
    raise AssertionError(name)


STEPS = [("sync", r"cluster\.sync\(\)"), ("form", r"\btied_runs\("), ("copy", r"R0->runs"),
         ("write", r"\bR\.runs\.(?:n|r\[0\]) ="), ("sort", r"\bquick_sort\("), ("give up", r"return false")]


def _steps(text):
    text = re.sub(r"//[^\n]*", "", text)
    found = [(m.start(), what) for what, pat in STEPS for m in re.finditer(pat, text)]
    return [what for _, what in sorted(found)]


def _path():
    """The steps of a block from the runs' forming to the sort of all boxes, whose first step is a barrier."""
    src = open(SRC).read()
    settle, split = _steps(_body(src, "settle_members")), _steps(_body(src, "split_boxes"))
    assert "form" in settle and "copy" in settle and "give up" in settle and "write" in split and split[-1] == "sort"
    return settle[:settle.index("give up")] + split[:-1] + ["sync"]


def _run(path, seed):
    rnd = random.Random(seed)
    runs, at = [None, None], [0] * BLOCKS   # two words of the first block's runs; each block's next step
    words = [0] * BLOCKS                    # words that a block has copied of them
    while any(k < len(path) for k in at):
        ready = [b for b in range(BLOCKS) if at[b] < len(path) and path[at[b]] != "sync"]
        if not ready:   # all at a barrier
            assert len(set(at)) == 1, "blocks at different barriers"
            at = [k + 1 for k in at]
            continue
        b = rnd.choice(ready)
        step = path[at[b]]
        if step == "copy":
            if b and runs[words[b]] != "tied":
                raise RuntimeError("a block copied runs that are not the batch's")
            words[b] += 1
            if words[b] < 2:
                continue
            words[b] = 0
        elif b == 0:
            runs = ["tied" if step == "form" else "all"] * 2
        at[b] += 1


def test_every_block_copies_the_runs_before_they_are_overwritten():
    for seed in range(200):
        _run(_path(), seed)


def test_a_missing_barrier_is_found():
    path = _path()
    copy = path.index("copy")
    cut = path[:copy + 1] + [s for s in path[copy + 1:-1] if s != "sync"] + ["sync"]
    with pytest.raises(RuntimeError):
        for seed in range(200):
            _run(cut, seed)
