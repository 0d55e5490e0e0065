"""Scattered lookups on the columns where the key start table, the searches
from a guess and the launch shape can go wrong, against the oracle: columns
of a few keys, sizes around a sector and a table group, runs of consecutive
keys, two scales of clusters (wide windows the guess misses), the extreme
keys, unaligned columns, and probe counts around a block and a launch-shape
threshold."""
import ctypes

import numpy as np
import pytest

from test_lookup_gpu import column, expected, from_dev_u32, probes_for, to_dev

pytestmark = pytest.mark.gpu

KINDS = ["binary_search", "btree", "harmonia", "radix_spline", "learned"]


def _columns(case, rng):
    if case == "tiny":
        for n in (1, 2, 3, 4, 5, 7, 8, 9, 31, 33, 63, 64, 65):
            yield column(rng, n)
    elif case == "run":
        yield np.arange(100, 100 + 4096, dtype=np.uint64)
        yield np.arange((1 << 64) - 5000, (1 << 64) - 1, dtype=np.uint64)
    elif case == "extremes":
        mid = column(rng, 4094)
        yield np.unique(np.concatenate([[0], mid, [(1 << 64) - 1]]).astype(np.uint64))
        yield np.array([0, (1 << 64) - 1], dtype=np.uint64)
    elif case == "two_scales":
        # clusters of clusters: every bucket holds either nothing or far too much
        big = np.sort(rng.choice(1 << 20, size=24, replace=False).astype(np.uint64)) << np.uint64(42)
        small = np.sort(rng.choice(1 << 16, size=64, replace=False).astype(np.uint64)) << np.uint64(14)
        fine = np.unique(rng.integers(0, 1 << 13, size=96, dtype=np.uint64))
        yield np.unique((big[:, None, None] + small[None, :, None] + fine[None, None, :]).ravel())
    else:  # "uniform"
        for n in (1023, 1024, 1025, 100_003):
            yield column(rng, n)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("case", ["tiny", "run", "extremes", "two_scales", "uniform"])
def test_scattered_lookups(orc, gj, cuda, case, kind, shift):
    import torch

    rng = np.random.default_rng(len(case) * 7 + len(kind))
    for col in _columns(case, rng):
        if kind == "harmonia":
            col = col[: len(col) // 32 * 32]
            if not len(col):
                continue
        pr = probes_for(rng, col, 3000)
        d = to_dev(torch, np.concatenate([np.zeros(4 - shift, dtype=np.uint64), col]))[4 - shift:]
        assert (d.data_ptr() % 32 == 0) == (shift == 0)
        ix = gj.make_index(kind).construct(None, d)
        np.testing.assert_array_equal(from_dev_u32(ix.lookup(to_dev(torch, pr))), expected(orc, kind, col, pr),
                                      err_msg=f"{len(col)} keys")


@pytest.mark.parametrize("kind", ["btree", "hash", "learned"])
@pytest.mark.parametrize("m", [255, 256, 257, 311_297, 16 * 152 * 8 * 256 - 1, 16 * 152 * 8 * 256 + 513])
def test_launch_shapes(orc, gj, cuda, kind, m):
    import torch

    rng = np.random.default_rng(m)
    col = column(rng, 40_000)
    pr = rng.choice(col, size=m)
    pr[::17] += np.uint64(1)
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    d_pr = to_dev(torch, pr)
    exp = expected(orc, kind, col, pr)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(d_pr)), exp)
    rows = torch.randperm(m, device="cuda").to(torch.int32)
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    ix.partitioned_lookup(d_pr, rows, out)
    np.testing.assert_array_equal(from_dev_u32(out)[rows.cpu().numpy()], exp)


@pytest.mark.parametrize("n", [1 << 14, 300_007])
@pytest.mark.parametrize("m", [(1 << 22) - 1, 1 << 22, (1 << 22) + 2049])
def test_long_unordered_spline_pairs(orc, gj, cuda, n, m):
    # the pairs kernel of eight probes a thread, at the size it starts from
    import torch

    rng = np.random.default_rng(n)
    col = column(rng, n)
    pr = probes_for(rng, col, m)[:m]
    ix = gj.radix_spline_index().construct(None, to_dev(torch, col))
    out, cnt = ix.inlj_pairs(to_dev(torch, pr), ordered=False)
    got = out[: 2 * int(cnt)].cpu().numpy().view(np.uint32).reshape(-1, 2)
    got = got[np.argsort(got[:, 0], kind="stable")]
    rows, pos = orc.pairs_from_positions(orc.bs_lookup(col, pr))
    np.testing.assert_array_equal(got[:, 0], rows)
    np.testing.assert_array_equal(got[:, 1], pos)


@pytest.mark.parametrize("kind,n", [("btree", (1 << 24) + 64), ("btree", 3 << 23), ("btree", (3 << 23) + 64),
                                    ("radix_spline", 300_007)])
@pytest.mark.parametrize("m", [(1 << 24) - 1, (1 << 25) + 2049])
def test_long_calls_through_nodes_and_splines(orc, gj, cuda, kind, n, m):
    # lookups, ordered pairs and partitioned lookups around the sizes from which
    # a thread takes several probes (tree nodes above 2^24 keys, splines)
    import torch

    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    col, pr = keys.cpu().numpy().view(np.uint64), probes.cpu().numpy().view(np.uint64)
    exp = (orc.exact_lookup if kind == "btree" else orc.bs_lookup)(col, pr)
    ix = gj.make_index(kind).construct(None, keys)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(probes)), exp)
    least = ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(least))
    ws = torch.full((least.value,), 0xA5, dtype=torch.uint8, device="cuda")
    out, cnt = ix.inlj_pairs(probes, workspace=ws)
    ix.inlj_pairs_status(ws, m)
    rows, pos = orc.pairs_from_positions(exp)
    got = out[: 2 * int(cnt)].cpu().numpy().view(np.uint32).reshape(-1, 2)
    np.testing.assert_array_equal(got[:, 0], rows)
    np.testing.assert_array_equal(got[:, 1], pos)
    rel = gj.range_partition(probes, int(keys[0]), 63 - 8, 8)
    scattered = torch.empty(m, dtype=torch.int32, device="cuda")
    ix.partitioned_lookup(rel.keys, rel.rows, scattered)
    np.testing.assert_array_equal(from_dev_u32(scattered), exp)


@pytest.mark.parametrize("hidden", [16, 32])
@pytest.mark.parametrize("n,m", [((1 << 23) + 32, (1 << 22) + 77), ((1 << 24) + 64, 5_000_011)])
def test_long_calls_through_network_roots(orc, gj, cuda, hidden, n, m):
    # learned indexes with an MLP root: several probes a thread from 16 waves of
    # a full chip on, whatever the column, and windows halved on any column
    import torch

    keys = gj.generate_sorted_keys(n, gj.DIST_LOGNORMAL, 1 << 63, seed=5)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    exp = orc.bs_lookup(keys.cpu().numpy().view(np.uint64), probes.cpu().numpy().view(np.uint64))
    ix = gj.make_index("learned", learned_root=gj.LEARNED_ROOT_MLP, learned_hidden=hidden,
                       learned_steps=20).construct(None, keys)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(probes)), exp)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup_sorted(probes)), exp)
    rel = gj.range_partition(probes, int(keys[0]), 55, 8)
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    ix.partitioned_lookup(rel.keys, rel.rows, out)
    np.testing.assert_array_equal(from_dev_u32(out), exp)


@pytest.mark.parametrize("W,L", [(4, 4), (7, 4), (8, 8), (15, 8), (16, 16), (32, 8), (64, 32)])
@pytest.mark.parametrize("n", [4096, 300_007, (1 << 24) + 64])
def test_long_calls_stage_tree_levels(orc, gj, cuda, W, L, n):
    # node formats without a key start table: blocks of several probes a thread
    # stage the upper levels, those of one search without them -- whole trees in
    # shared memory, and the top of larger ones
    import torch

    m = 5_000_011
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    exp = orc.exact_lookup(keys.cpu().numpy().view(np.uint64), probes.cpu().numpy().view(np.uint64))
    ix = gj.btree_index(btree_node_keys=W, btree_leaf_keys=L).construct(None, keys)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(probes)), exp)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(probes[:1001])), exp[:1001])
    rel = gj.range_partition(probes, int(keys[0]), 55, 8)
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    ix.partitioned_lookup(rel.keys, rel.rows, out)
    np.testing.assert_array_equal(from_dev_u32(out), exp)
    rows, pos = orc.pairs_from_positions(exp)
    for ordered in (True, False):
        prs, cnt = ix.inlj_pairs(probes, ordered=ordered)
        got = prs[: 2 * int(cnt)].cpu().numpy().view(np.uint32).reshape(-1, 2)
        if not ordered:
            got = got[np.argsort(got[:, 0], kind="stable")]
        np.testing.assert_array_equal(got[:, 0], rows)
        np.testing.assert_array_equal(got[:, 1], pos)


@pytest.mark.parametrize("m", [1, (1 << 18) - 1, 1 << 18, (1 << 18) + 2049])
def test_fence_in_host_memory(orc, gj, cuda, m):
    # a binary search whose sampled keys lie in host memory: lookups, ordered
    # pairs (two passes) and partitioned lookups around the size of long blocks
    import torch

    rng = np.random.default_rng(m)
    col = column(rng, 70_001)
    pr = probes_for(rng, col, m)[:m]
    exp = orc.bs_lookup(col, pr)
    ix = gj.binary_search_index(index_memory=gj.INDEX_MEMORY_HOST).construct(None, to_dev(torch, col))
    d_pr = to_dev(torch, pr)
    np.testing.assert_array_equal(from_dev_u32(ix.lookup(d_pr)), exp)
    prs, cnt = ix.inlj_pairs(d_pr)
    got = prs[: 2 * int(cnt)].cpu().numpy().view(np.uint32).reshape(-1, 2)
    rows, pos = orc.pairs_from_positions(exp)
    np.testing.assert_array_equal(got[:, 0], rows)
    np.testing.assert_array_equal(got[:, 1], pos)
    rel = gj.range_partition(d_pr, int(col[0]), 55, 8)
    out = torch.empty(m, dtype=torch.int32, device="cuda")
    ix.partitioned_lookup(rel.keys, rel.rows, out)
    np.testing.assert_array_equal(from_dev_u32(out), exp)
