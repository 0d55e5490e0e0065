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


@pytest.fixture
def start_tables(gj):
    """limit(bytes): key start tables above it find no memory; returns the
    tables built since the last call."""
    limit = gj.lib().gj_debug_start_tables
    limit(2**64 - 1)
    yield limit
    limit(2**64 - 1)


@pytest.mark.parametrize("limit", [0, 20_000_000])
@pytest.mark.parametrize("kind,n", [("btree", 1_000_000), ("btree", (1 << 25) + 64), ("harmonia", 1 << 20),
                                    ("binary_search", (1 << 25) + 64), ("radix_spline", (1 << 25) + 64)])
def test_full_device_builds_without_tables(gj, cuda, start_tables, kind, n, limit):
    # no memory for any table, or none for the finer one of large ordered
    # pairs: the index is built, and gives what it gives with them
    import torch

    m = (1 << 25) + 257
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    ix = gj.make_index(kind).construct(None, keys)
    full = start_tables(limit)
    assert full == (2 if n > 1 << 24 else 1)
    short = gj.make_index(kind).construct(None, keys)
    assert start_tables(2**64 - 1) == (0 if limit == 0 else 1)
    assert short.memory_consumption() < ix.memory_consumption() or full == 1 and limit > 0
    assert torch.equal(short.lookup(probes), ix.lookup(probes))
    (pairs, count), (short_pairs, short_count) = ix.inlj_pairs(probes), short.inlj_pairs(probes)
    assert int(count) == int(short_count)
    assert torch.equal(pairs[: 2 * int(count)], short_pairs[: 2 * int(count)])


def test_learned_root_choice_builds_its_table_once(gj, cuda, start_tables):
    # four roots are built and three thrown away; the table of ordered pairs
    # (its coarse and its finer form) depends on the column alone
    keys = gj.generate_sorted_keys((1 << 25) + 64, gj.DIST_UNIFORM, 1 << 63, seed=5)
    gj.make_index("learned", learned_steps=20).construct(None, keys)
    assert start_tables(2**64 - 1) == 2
