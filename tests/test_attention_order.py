"""The attention kernels' forms: which launches take which, and the order of the backward walk's bulk operations on the
dQ sums (host rules and a replay, no GPU needed)."""
import ctypes

import pytest

from allie_b200.ops import _lib

pytestmark = pytest.mark.skipif(not _lib.have_cuda_lib(), reason="kernel library not built")

STORE, ADD, READ, DQ_OUT, DKV_OUT = range(5)


@pytest.mark.parametrize("nt", list(range(1, 13)) + [32])
def test_every_sum_waits_for_what_it_builds_on(nt):
    """Bulk groups of a thread complete in any order unless it waits: with as many of the latest under way as the
    waits allow, whatever touches the sum of a query tile finds everything before it on that tile complete."""
    room = 8192
    buf, slices = (ctypes.c_int * (4 * room))(), 3
    n = _lib.cuda().ab_attn_bwd_walk_order(nt, slices, buf, room)
    assert 0 < n <= room
    open_groups, content, adds = [], {}, 0          # tiles of the groups under way; contributions per tile
    for i in range(n):
        what, slice_, tile, may_be_open = buf[4 * i:4 * i + 4]
        if may_be_open >= 0:
            open_groups = open_groups[len(open_groups) - may_be_open:] if may_be_open else []
        if what in (STORE, ADD, READ):
            assert tile not in open_groups, (i, what, slice_, tile)
        if what == STORE:
            content[tile] = [slice_]
        elif what == ADD:
            assert content[tile] and set(content[tile]) == {slice_}
            content[tile].append(slice_)
            adds += 1
        elif what == READ:                          # all key tiles before the query tile have contributed
            assert content.pop(tile) == [slice_] * tile
        if what != READ:
            open_groups.append(tile if what in (STORE, ADD) else None)
    assert adds == slices * (nt - 1) * (nt - 2) // 2
    assert content == {tile: [slices] for tile in range(1, nt)}


@pytest.mark.parametrize("slices,T,walks", [
    (1, 128, 1), (4, 256, 1), (16, 128, 1), (16, 256, 1), (16, 384, 0), (20, 384, 0), (16, 512, 0), (32, 512, 0), (48, 512, 1),
    (32, 640, 0), (48, 640, 1), (32, 1024, 0), (148, 1024, 1), (200, 1000, 1), (320, 128, 1), (1024, 512, 1),
])
def test_the_form_that_measured_faster(slices, T, walks):
    """Sizes at which one form of the backward beats the other by more than 3 % on a GPU of 148 SMs."""
    assert _lib.cuda().ab_attn_bwd_walks(slices, T, 148) == walks


@pytest.mark.parametrize("hd,tiles,least", [(64, 1, 297), (64, 2, 297), (64, 3, 445), (64, 4, 593), (64, 8, 1185),
                                            (128, 1, 593), (128, 4, 593), (128, 8, 1185)])
def test_launches_of_few_items_keep_a_block_per_item(hd, tiles, least):
    rule = _lib.cuda().ab_attn_fwd_takes_over
    assert rule(least, tiles, hd, 148) == 1
    assert all(rule(n, tiles, hd, 148) == 0 for n in (1, 16, 296, least - 1))
