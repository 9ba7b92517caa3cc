"""How the blocks of a row arrive at their meetings (csrc/split_kernel.cuh), by reading: what a wrong
order costs is a race on shared memory, which no launch is made to show."""
import os
import re

CSRC = os.path.join(os.path.dirname(__file__), "..", "lily-qwen3.8-flash-next_b200", "csrc")


def _body(source, name):
    at = re.search(r"\b%s\([^;{]*\)\s*\{" % name, source)
    assert at, name
    depth, end = 1, at.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(source[end], 0)
        end += 1
    return source[at.end():end]


def test_the_lists_meeting_releases_what_the_block_has_read():
    # A block that has met the others with its list stores into the first block's `best_of`: the first
    # block's own reads of that memory (marks, runs of its list) have to come before.
    with open(os.path.join(CSRC, "split_kernel.cuh")) as f:
        source = f.read()
    merge = _body(source, "merge_lists")
    arrivals = re.findall(r"(arrive\w*)\((?:list_bar|peer_smem\(&ss->mbar\[MEET_LISTS\])", merge)
    assert arrivals and "peer_smem(best_of + place, 0)" in merge
    # (The runs lie elsewhere: they are read behind the arrival.)
    assert not re.search(r"run_of = [^;]*best_of", merge)
    for name in arrivals:
        body = _body(source, name)
        assert "mbarrier.arrive." in body and ".release.cluster." in body, name


def test_no_list_of_buckets_lies_where_a_late_block_may_store():
    # `flagged` lies over `tmax`, into which the other blocks of a wide row put their maxima. A block whose wait for
    # them ran out goes on to the later meetings, but its list counts as full: nothing is written to it or read
    # from it. (Nothing but the list's own adds changes its length after that.)
    with open(os.path.join(CSRC, "split_args.cuh")) as f:
        union = re.search(r"union \{(.*?)\n    \};", f.read(), re.S).group(1)
    assert "flagged[" in union and "tmax[" in union
    with open(os.path.join(CSRC, "split_kernel.cuh")) as f:
        source = f.read()
    wait = source.index("wait_first_phase(&ss->mbar[MEET_POOL], ca.wait_ns >> 2)", source.index("ss->bin = NONE;"))
    out = source[wait:source.index("spl_sync();", wait)]
    assert "ss->hard = ss->late = 1;" in out and "ss->n_flagged = SPL_FLAGGED + 1u;" in out
    listed = source.index("atomicAdd(&ss->n_flagged", wait)
    assert not re.search(r"n_flagged\s*=[^=]", source[wait + len(out):listed])
    write = source.index("ss->flagged[at++] =", listed)
    assert "at < SPL_FLAGGED" in source[listed:write]
    refuse = source.index("if (n_flagged > SPL_FLAGGED) {", write)
    assert refuse < source.index("ss->flagged[i / SPL_U]", refuse)
    assert source.count("ss->flagged[") == 2
