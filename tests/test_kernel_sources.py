"""What a kernel's source has to keep and no run on one GPU can be relied on to show."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tnn_b200", "csrc")


def _enclosing_block(text, at):
    """The innermost { ... } around position `at`."""
    depth, i = 0, at
    while depth >= 0:
        i -= 1
        depth += {"}": 1, "{": -1}.get(text[i], 0)
    depth, j = 1, i
    while depth:
        j += 1
        depth += {"{": 1, "}": -1}.get(text[j], 0)
    return text[i:j + 1]


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu"))))
def test_every_commit_stands_with_the_umma_it_covers(name):
    """tcgen05.commit covers the UMMAs of the thread that executes it, and no other's.  Where one elected lane issues the
    UMMAs, a commit under `lane == 0` beside that block may come from another lane and complete at once: the barrier
    would hand a shared-memory stage back while a UMMA still reads it.  So every commit is in the block of its UMMAs."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"\bumma_commit(_pair)?\(&?\w", text):
        block = _enclosing_block(text, m.start())
        assert re.search(r"\bumma_f16_\w+\(", block), text[max(0, m.start() - 120):m.end() + 40]
