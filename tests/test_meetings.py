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
    # them ran out goes on to the later meetings, but has no bound: it is `hopeless`, and lists and reads nothing.
    with open(os.path.join(CSRC, "split_args.cuh")) as f:
        union = re.search(r"union \{(.*?)\n    \};", f.read(), re.S).group(1)
    assert "flagged[" in union and "tmax[" in union
    with open(os.path.join(CSRC, "split_kernel.cuh")) as f:
        source = f.read()
    wait = source.index("wait_first_phase(&ss->mbar[MEET_POOL], ca.wait_ns >> 2)", source.index("ss->bin = NONE;"))
    bound = re.search(r"bound_key = ([^;]*?)\? 0u", source[wait:])
    assert re.search(r"\{\s*ss->hard = ss->late = 1;", source[wait:wait + 200])
    assert "ss->late != 0u" in bound.group(1)
    # (The barrier between the two makes it one value for all threads: other blocks' waits set their own.)
    assert "spl_sync();" in source[wait:wait + bound.start()]
    hopeless = source.index("const bool hopeless = bound_key == 0u", wait)
    assert hopeless < source.index("if (hopeless) {", hopeless) < source.index("ss->flagged[at++]", hopeless)
