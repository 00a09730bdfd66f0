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


def test_the_wait_for_an_item_outlasts_the_longest_one():
    """The item warp of the dQ kernel waits through a whole item, up to 2^25 K/V rows in tiles of 64 that take some 1200 cycles."""
    text = code("range_dense.cu")
    wait = re.search(WAIT + r"&it_empty\[n % kDqItems\][^;]*;", text).group(0)
    more = re.search(r"FSA_WAIT_CLOCKS \+ longest \* kDqTileClocks", wait) and int(re.search(r"kDqTileClocks = (\d+)", text).group(1))
    least = int(re.search(r"define FSA_WAIT_CLOCKS (\d+)u", open(os.path.join(CSRC, "sm100_prims.cuh")).read()).group(1))
    assert (1 << 25) // 64 * 1200 < least + (1 << 25) // 64 * (more or 0) < 1 << 32
    assert re.search(r"longest = max\(longest, m\.nblk\)", text)


def test_a_failed_launch_of_several_problems_says_so_in_the_words_of_all():
    """A CTA of range_fwd_dense takes over items of any problem: one that gave up has left work of each of them undone."""
    text = code("range_dense.cu")
    kernel = text[text.index("range_fwd_dense(const") : text.index("static cudaError_t launch_rd")]
    assert set(re.findall(WAIT + r"[^;]*?, (status), limit\)", kernel)) == {"status"} and re.search(r"int\* status = reinterpret_cast<int\*>\(bars", kernel)
    assert "*status = kStatusOk;" in kernel[: kernel.index("__syncthreads")]
    assert re.search(r"__syncthreads\(\);[^}]*if \(tid < kRdProblems && \*status != kStatusOk && launch\.p\[tid\]\.status\) atomicMax", kernel)


COLLECTIVE = r"tmem_ld|tmem_st|_sync\(|__syncwarp|__syncthreads|warp_ok|warp_stays|bar_all|bar\.sync"
VOTE = r"warp_ok\(|warp_stays\(|bar_all\(|__syncthreads_and\(|= __shfl_sync\(0xffffffffu, ok "


def closing(text, at):
    """The place behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] in "({[") - (text[i] in ")}]")
        if depth == 0:
            return i + 1
    raise ValueError("unbalanced")


def inlined(text):
    """The lambdas that wait or vote in the place of their calls."""
    while True:
        for m in re.finditer(r"auto (\w+) = \[&\]\([^)]*\)\s*\{", text):
            end = closing(text, m.end() - 1)
            body = text[m.end() - 1 : end]
            if re.search(WAIT + "|" + VOTE, body):
                break
        else:
            return text
        rest = re.sub(r"(?<![\w.])" + m.group(1) + r"\((?=[^)]*\))", lambda c: body.replace("return", "") + " (", text[end + 1 :])
        text = text[: m.start()] + rest


def lanes_apart(text):
    """Walks a source in order, a loop's body twice: the loops in which lanes meet, but which a lane whose wait ran out may leave alone."""
    loops = []
    events = re.compile(r"(?P<loop>(?:for|while) \()|(?P<vote>" + VOTE + r")|(?P<wait>" + WAIT + r")|(?P<leave>if \([^()]*!ok[^()]*\) (?:break|continue))"
                        r"|(?P<other>\} else (?:if \(warp|\{\s*(?:if \(warp|bool ok|const int)))|(?P<fresh>bool ok(?:_wait)? = true)")

    def walk(a, b, apart, owner):
        """apart: lanes may differ on whether a wait ran out; owner: the innermost loop, whether lanes meet in it."""
        while True:
            m = events.search(text, a, b)
            if not m:
                return apart
            a = m.end()
            if m.group("vote"):
                apart = False
            elif m.group("wait"):
                apart = True
            elif m.group("fresh") or m.group("other"):
                apart = False
            elif m.group("leave"):
                if apart and owner and owner[1]:
                    loops.append(owner[0])
            else:
                head_end = closing(text, m.end() - 1)
                head = text[m.start() : head_end]
                brace = re.compile(r"\s*\{").match(text, head_end)
                if not brace:
                    continue
                end = closing(text, brace.end() - 1)
                me = (head, re.search(COLLECTIVE, head + text[head_end:end]) is not None)
                for _ in range(2):
                    if "warp_stays" in head:
                        apart = False
                    elif re.search(r"\bok\b|ok_wait", head) and me[1] and apart:
                        loops.append(head)
                    apart = walk(brace.end(), end, apart, me)       # (a loop that ends by its count ends without the vote in its head)
                a = end

    walk(0, len(text), False, None)
    return loops


@pytest.mark.parametrize("name", SOURCES)
def test_lanes_leave_a_loop_in_which_they_meet_together(name):
    assert not lanes_apart(inlined(code(name)))


@pytest.mark.parametrize("name,votes", [("range_dense.cu", ["scale_acc", "all_visible"]), ("sel_fwd.cu", ["masked"]), ("sel_bwd_pipe.cu", ["all_visible"])])
def test_a_vote_that_stands_for_the_loops_counts_the_lanes_that_gave_up(name, votes):
    """Where a warp votes in each turn for another reason, that vote tells too whether one on the waits is due."""
    text = code(name)
    for v in votes:
        m = re.search(r"const bool " + v + r" = __(?:any_sync\(0xffffffffu, [^;]*\|\| !ok|all_sync\(0xffffffffu, ok &&[^;]*)\);", text)
        assert m and re.match(r"\s*if \((?:" + v + r"\) \{\s*ok = ok && [^;]*;\s*if \(!warp_stays|!?" + v + r" && !warp_stays)\(ok\)\) break;", text[m.end():]), v
