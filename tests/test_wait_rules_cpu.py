"""Rules of the kernels' waits that a run cannot show (a breach needs a lane that is late by microseconds), read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "flash-sparse-attention_b200", "csrc")
SOURCES = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")))
WAIT = r"mbar_(?:wait|poll)\w*\("


def code(name):
    """The source without comments."""
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def line(text, at):
    return text.count("\n", 0, at) + 1


@pytest.mark.parametrize("name", SOURCES)
def test_a_warp_meets_between_its_waits_and_what_one_lane_issues(name):
    text = code(name)
    waits = [m.end() for m in re.finditer(WAIT, text)]
    meets = [m.start() for m in re.finditer(r"warp_ok\(|__syncwarp\(", text)]
    alone = [m.start() for m in re.finditer(r"if \((?:ok && )?(?:leader|lane == 0)\) (?:\{\s*(?:s_item|s_rec|#pragma|constexpr|const uint32_t|umma)|mbar_arrive)", text)]
    for at in alone:
        last = max((w for w in waits if w < at), default=None)
        assert last is None or any(last < m < at for m in meets), f"{name}:{line(text, at)}"
