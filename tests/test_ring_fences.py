"""The candidate ring between a screening and a rescoring warp of the tensor-core search: one lane acquires
the other warp's counter, and a shuffle, which hands the value to the other lanes, orders no memory.  Checked
in the source: every poll goes through the one helper that ends in a warp barrier, and every release
follows one."""
import os
import re

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'nngpr_b200', 'csrc',
                        'knn_tc.cu')).read()


def body(name):
    """(start, end) of the function defined as `name(...) {...}`."""
    start = re.search(r'\b%s\([^;{]*\{' % name, SRC).end()
    depth, j = 1, start
    while depth:
        depth += {'{': 1, '}': -1}.get(SRC[j], 0)
        j += 1
    return start, j


def calls(name):
    return [m.start() for m in re.finditer(r'\b%s\(' % name, SRC)]


def test_an_acquire_reaches_the_other_lanes_through_a_barrier():
    a, b = body('warp_poll')
    code = SRC[a:b]
    assert code.rindex('__syncwarp()') > code.rindex('__shfl_sync(') > code.index('poll_bounded(')
    inside = [c for c in calls('poll_bounded') if a < c < b]
    assert len(inside) == 1 and len(calls('poll_bounded')) == 2  # the definition, and the helper's call
    pa, pb = body('poll_bounded')
    assert all(pa < c < pb for c in calls('ld_acquire')[1:])
    assert len(calls('warp_poll')) == 3  # the definition, for places, for entries


def test_a_release_follows_a_barrier():
    releases = calls('st_release')[1:]
    assert len(releases) == 3
    for c in releases:
        before = SRC[:c]
        # nothing but the owner's own bookkeeping between the barrier and lane 0's store
        between = before[before.rindex('__syncwarp();') + len('__syncwarp();'):]
        assert re.fullmatch(r'\s*(tail \+= cnt;\s*)?if \(lane == 0\) ', between), between
