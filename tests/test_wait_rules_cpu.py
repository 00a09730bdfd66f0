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


@pytest.mark.parametrize("name", SOURCES)
def test_a_wait_that_ran_out_is_a_roles_last(name):
    text = code(name)
    late = [line(text, m.start()) for m in re.finditer(WAIT + r"[^;]*\)\s*&&\s*ok\b", text)]
    assert not late, f"{name}: lines {late} wait before they look whether an earlier wait ran out"


def test_what_is_issued_depends_on_the_wait_before_it():
    """A tensor copy or product whose wait ran out would be in flight when the CTA ends, or take its place from numbers nobody has written."""
    for name in SOURCES:
        text = code(name)
        for m in re.finditer(r"ok = (?:ok && )?" + WAIT + r"[^;]*;", text):
            rest = text[m.end():]
            first = re.search(r"tma_load|tma_store|umma_ss|umma_ts|issue_mma", rest)
            again = re.search(WAIT, rest)
            if first and (again is None or first.start() < again.start()):
                assert re.search(r"if \(!ok\)|if \(ok\)|if \(tid == 0 && ok\)|&& ok;|\bok &&", rest[: first.start()]), f"{name}:{line(text, m.start())}"


@pytest.mark.parametrize("name,writes,reads,barrier", [
    ("sel_fwd.cu", "umma_ss(d_s", "umma_ts(d_o", "s_empty"),
    ("range_dense.cu", "umma_ss(tbase + cS", "umma_ts(tbase + cO", "pv_done"),
    ("range_dense.cu", "umma_ts(tbase + b * 128 + BK, tbase + cDO", "umma_ts(tbase + cDQ", "ds_empty"),
    ("range_bwd_dkdv.cu", "umma_ss(c_s", "umma_ts(c_acc", "in_read"),
])
def test_a_product_waits_for_the_one_that_reads_what_it_overwrites(name, writes, reads, barrier):
    """Products of one thread run in the order of their issue only where accumulator and shape are the same; a commit tells when one is done."""
    text = code(name)
    assert text.count(writes) == 1 and text.count(reads) == 1
    before = text[: text.index(writes)]
    waits = list(re.finditer(WAIT + r"&" + barrier + r"\[", before))
    assert waits and "umma_" not in before[waits[-1].end():].replace("umma_desc", "").replace("umma_idesc", ""), f"{name}: {writes}"
    after = text[text.index(reads):]
    commit = re.search(r"umma_commit\(&" + barrier + r"\[", after)
    assert commit and "mbar_" not in after[: commit.start()], f"{name}: {reads}"
