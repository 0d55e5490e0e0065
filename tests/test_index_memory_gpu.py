"""Device memory of an index: what it holds is what it reports, and a key start
table that none of its calls reads is not kept."""
import pytest

pytestmark = pytest.mark.gpu


def held(torch, build):
    """(index, device bytes its build left allocated)"""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    ix = build()
    torch.cuda.synchronize()
    return ix, before - torch.cuda.mem_get_info()[0]


def test_unread_start_table_is_given_back(gj, cuda):
    # evenly spread keys above 2^24: lookups search the nodes, and ordered pairs
    # are not partitioned below 3 * 2^23 keys
    keys = gj.generate_sorted_keys(20_000_000, gj.DIST_UNIFORM, 1 << 63, seed=5)
    nodes_only = gj.btree_index(btree_start_bits=18).construct(None, keys).memory_consumption()
    assert gj.btree_index().construct(None, keys).memory_consumption() == nodes_only


@pytest.mark.parametrize("kind", ["btree", "radix_spline"])
def test_unaligned_column_keeps_no_table_for_pairs(gj, cuda, kind):
    # pairs into a column off the sector boundary are never partitioned: no
    # table is kept for them (2^24 entries beside the aligned column's index)
    keys = gj.generate_sorted_keys((1 << 25) + 65, gj.DIST_UNIFORM, 1 << 63, seed=5)
    aligned = gj.make_index(kind).construct(None, keys[:-1]).memory_consumption()
    unaligned = gj.make_index(kind).construct(None, keys[1:]).memory_consumption()
    assert aligned - unaligned > 60_000_000


@pytest.mark.parametrize("kind,dist,n", [("btree", "DIST_CLUSTERS", (1 << 27) + 64), ("btree", "DIST_UNIFORM", 1 << 27),
                                         ("btree", "DIST_UNIFORM", 20_000_000), ("harmonia", "DIST_CLUSTERS", 1 << 26)])
def test_held_is_reported(gj, cuda, kind, dist, n):
    import torch

    small = gj.btree_index().construct(None, gj.generate_sorted_keys(1 << 16, 0, 1 << 63, seed=1))  # pools are warm
    keys = gj.generate_sorted_keys(n, getattr(gj, dist), 1 << 63, seed=5)
    ix, bytes_held = held(torch, lambda: gj.make_index(kind).construct(None, keys))
    reported = ix.memory_consumption()
    # allocations come in steps of 2 MB, a handful an index
    assert reported - (2 << 20) <= bytes_held <= reported + (8 << 20), (bytes_held, reported)
    del small
