"""What the blocks of a cluster solve (rbsor_cluster.cu) owe one another, read
from its source: a broken order here shows as a wrong iterate or a GPU fault once
in many runs, so it is not provoked on a GPU."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = open(os.path.join(ROOT, "paintop_b200", "csrc", "rbsor_cluster.cu")).read()


def _body(head):
    """The content of the brace that `head` opens."""
    at = SOURCE.index(head)
    i = start = at + head.index("{") if "{" in head else SOURCE.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(SOURCE[i], 0)
        i += 1
        if depth == 0:
            return SOURCE[start + 1:i - 1]


def _branches():
    """The workers' branches that show rows by plain stores: the re-run's and the fold's."""
    return [_body("else if (mode == M_REDO) {"), _body("} else {  // M_FOLD")]


def test_plain_row_stores_lie_between_two_meetings():
    """show(h, false) stores plainly where asynchronous stores of the step before
    may still be landing; the meeting before it waits for those, the one after
    for the rows themselves."""
    for body in _branches():
        calls = re.findall(r"cluster_meet\(\)|show\(\d, (?:true|false)\)|sweeps\(|near\(", body)
        shows = [k for k, c in enumerate(calls) if c.startswith("show")]
        assert shows and all(c.endswith("false)") for c in calls if c.startswith("show"))
        assert calls[shows[0] - 1] == "cluster_meet()" and shows[0] > 0, calls
        assert calls[shows[-1] + 1] == "cluster_meet()", calls


def test_the_books_meet_as_often_as_the_workers():
    books = _body("if (mode != M_SWEEP) {")
    for body in _branches():
        assert books.count("cluster_meet()") == body.count("cluster_meet()")


def test_the_hardware_barrier_pairs_only_starts_and_ends():
    """barrier.cluster is anonymous: a block that gave up a wait and leaves must not
    pair with another's re-run or fold. So a thread takes it once before its first
    bounded wait and once in leave()."""
    region = _body("__device__ __forceinline__ void solve_region(")
    assert region.count("cluster_sync()") == 1
    assert region.index("cluster_sync()") < region.index("keep_books(")
    assert "cluster_sync()" not in _body("__device__ __forceinline__ void keep_books(")
    leave = _body("__device__ __forceinline__ void leave(")
    assert leave.count("cluster_sync()") == 1 and SOURCE.count("barrier.cluster.arrive") == 1
    # every way out after the first barrier is leave(), except for warps without patches before it counts them
    rest = region[region.index("cluster_sync()"):]
    ends = re.findall(r"leave\(P\);\s*(?:return;|$)", rest.rstrip())
    assert len(ends) == 2
