"""The partitioned INLJ's directory on the columns that stress it, against
the oracle: a column whose keys crowd into a few buckets (long lower-bound
ranges, searched past the first sectors), a column that is not 32-byte
aligned, columns of a few keys, clustered keys with long gaps (buckets
filled by the prefix maximum), narrower key ranges, a run of consecutive
keys, probes outside the key range, several windows, and the directory
built per call or kept with the index.
Positions must equal the oracle's per probe row, the pairs as a set (their
order across tiles is not fixed)."""
import ctypes

import numpy as np
import pytest

from test_lookup_gpu import column, expected, from_dev_u32, probes_for, to_dev

pytestmark = pytest.mark.gpu

KINDS = ["btree", "binary_search", "radix_spline", "hash", "learned", "no_op"]


def _column(case, rng):
    if case == "wide":
        # 2^19 dense keys in partition 0 (2^17 sectors: too wide for the
        # directory) and 2^19 keys spread over the rest of the range
        dense = np.arange(1000, 1000 + (1 << 19), dtype=np.uint64)
        sparse = np.unique(rng.integers(1 << 40, 1 << 63, size=(1 << 19) + 4096, dtype=np.uint64))[: 1 << 19]
        return np.concatenate([dense, sparse])
    if case == "clusters":
        starts = np.sort(rng.choice(1 << 50, size=64, replace=False).astype(np.uint64)) << np.uint64(10)
        col = np.concatenate([s + np.arange(4096, dtype=np.uint64) * np.uint64(3) for s in starts])
        return np.unique(col)
    if case == "tiny":
        return np.array([5, 17, 1 << 40, (1 << 64) - 2, (1 << 64) - 1], dtype=np.uint64)
    # narrower key ranges (directory buckets a few keys wide), and a run of
    # 3000 consecutive keys inside one bucket among sparse ones
    if case == "range48":
        return column(rng, 100_003, upper=1 << 48)
    if case == "range52":
        return column(rng, 1 << 17, upper=1 << 52)
    if case == "run":
        col = column(rng, 1 << 17, upper=1 << 49)
        return np.unique(np.concatenate([col, np.arange(1 << 40, (1 << 40) + 3000, dtype=np.uint64)]))
    return column(rng, 100_003)  # "unaligned" and "plain"


@pytest.mark.parametrize("prepared", [False, True])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("case", ["wide", "unaligned", "tiny", "clusters", "range48", "range52", "run"])
def test_partitioned_directory_cases(orc, gj, cuda, kind, case, prepared):
    import torch

    rng = np.random.default_rng(len(case) * 31 + len(kind))
    col = _column(case, rng)
    pr = probes_for(rng, col, 60_000)
    if case == "unaligned":
        d_all = to_dev(torch, np.concatenate([np.array([0], dtype=np.uint64), col]))
        d_col = d_all[1:]  # 8-byte offset: not 32-byte aligned
        assert d_col.data_ptr() % 32 != 0
    else:
        d_col = to_dev(torch, col)
    ix = gj.make_index(kind).construct(None, d_col)
    if prepared:  # the directory kept with the index instead of built per call
        ix.prepare_partitioned()
    exp = expected(orc, kind, col, pr)
    erows, epos = orc.pairs_from_positions(exp)
    # the wide scatter (fanout 2^8 and up), the narrow one (below 2^8), and the
    # default fanout (0: about 2^20 keys a partition, from 2^5)
    for bits, window in ((8, 0), (12, 0), (10, 7777), (5, 0), (6, 20000), (0, 0)):
        pos, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=bits, positions=True,
                                            pairs=True)
        got = from_dev_u32(pos)
        bad = np.nonzero(got != exp)[0]
        assert len(bad) == 0, f"{kind}/{case}/2^{bits}: {len(bad)} positions differ, rows {bad[:5]}"
        c = int(cnt.item())
        a = prs[: 2 * c].cpu().numpy().view(np.uint32).reshape(-1, 2)
        order = np.argsort(a[:, 0], kind="stable")
        np.testing.assert_array_equal(a[order, 0], erows, err_msg=f"{kind}/{case}/2^{bits}")
        np.testing.assert_array_equal(a[order, 1], epos, err_msg=f"{kind}/{case}/2^{bits}")


@pytest.mark.parametrize("kind", ["btree", "binary_search"])
def test_partitioned_skewed_probes(orc, gj, cuda, kind):
    # Nearly every probe falls into one narrow key range (one partition, a
    # few directory buckets), every 64th into the lowest keys, some are
    # absent: one partition far fuller than the others, across windows.
    import torch

    rng = np.random.default_rng(77)
    col = column(rng, 1 << 18)
    m = 300_000
    hot = col[(1 << 17):(1 << 17) + 512]
    pr = hot[rng.integers(0, len(hot), m)]
    pr[::64] = col[rng.integers(0, 64, len(pr[::64]))]
    pr[::97] = pr[::97] + np.uint64(1)  # some absent keys
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    exp = expected(orc, kind, col, pr)
    erows, epos = orc.pairs_from_positions(exp)
    for prepared in (False, True):
        if prepared:
            ix.prepare_partitioned()
        for bits, window in ((8, 0), (11, 0), (8, 65536), (5, 0), (7, 65536)):
            pos, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=bits,
                                                positions=True, pairs=True)
            np.testing.assert_array_equal(from_dev_u32(pos), exp, err_msg=f"{kind}/2^{bits}/{window}")
            c = int(cnt.item())
            a = prs[: 2 * c].cpu().numpy().view(np.uint32).reshape(-1, 2)
            order = np.argsort(a[:, 0], kind="stable")
            np.testing.assert_array_equal(a[order, 0], erows)
            np.testing.assert_array_equal(a[order, 1], epos)


@pytest.mark.parametrize("radix_bits", range(1, 13))
@pytest.mark.parametrize("m", [1, 4095, 4096, 4097, 70_001, 2 * 152 * 8192 + 8191])
def test_range_partition_layout(gj, cuda, radix_bits, m):
    # the relation itself: partitions in key order, whole and disjoint, the
    # tuples of earlier tiles first, and every row id with its own key; both
    # tile sizes, every fanout (shared memory up to its limits)
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(radix_bits * 1000 + m)
    keys = torch.randint(0, 1 << 40, (m,), generator=g, device="cuda", dtype=torch.int64)
    keys[: m // 3] = keys[: m // 3] % 1000  # a crowded partition
    low, shift = 500, 40 - radix_bits
    rel = gj.range_partition(keys, low, shift, radix_bits)
    part = torch.clamp((keys - low).clamp(min=0) >> shift, max=(1 << radix_bits) - 1)
    sizes = torch.bincount(part, minlength=1 << radix_bits)
    assert int(rel.offsets[0]) == 0 and torch.equal(rel.offsets[1:], torch.cumsum(sizes, 0))
    rows = rel.rows.to(torch.int64)
    assert torch.equal(torch.sort(rows)[0], torch.arange(m, device="cuda"))
    assert torch.equal(keys[rows], rel.keys)
    assert torch.equal(part[rows], torch.sort(part)[0])
    tile = rows // 8192  # chunks of whole tiles of either size come in order
    order = part[rows] * (1 << 20) + tile
    assert bool((order[1:] >= order[:-1]).all())


@pytest.mark.parametrize("radix_bits", [1, 5, 7, 8, 11, 12])
@pytest.mark.parametrize("m,window", [((1 << 22) + 1, 0), (3 * (1 << 22) - 77, 1 << 22)])
def test_positions_through_the_inverse(orc, gj, cuda, radix_bits, m, window):
    # windows large enough for the gather pass that brings positions back to
    # probe order (the last, shorter window stores them by row): one ragged
    # window and several, through both scatter kernels, and a fanout whose
    # runs do not fit beside the offsets
    import torch

    rng = np.random.default_rng(radix_bits)
    col = column(rng, 300_007)
    pr = probes_for(rng, col, m)[:m]
    # kinds whose plain lookup is not taken for windows of this size, and one for which it is
    for kind, params in (("radix_spline", {}), ("btree", {"btree_node_keys": 8}), ("btree", {})):
        ix = gj.make_index(kind, **params).construct(None, to_dev(torch, col)).prepare_partitioned()
        got, _, _ = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=radix_bits)
        np.testing.assert_array_equal(from_dev_u32(got), expected(orc, kind, col, pr))


@pytest.mark.parametrize("kind,window,m,bits,pairs", [("btree", 1_300_000, 2_500_000, 0, True),
                                                      ("hash", 1_500_000, 2_700_000, 5, True),
                                                      ("radix_spline", 5_000_000, 9_900_000, 0, False),
                                                      ("btree", 2_600_000, 5_050_000, 11, True)])
def test_uneven_windows(orc, gj, cuda, kind, window, m, bits, pairs):
    # a last window a little shorter than the others, whose tiles form more
    # chunks than a whole window's
    import torch

    rng = np.random.default_rng(m)
    col = column(rng, 300_007)
    pr = probes_for(rng, col, m)[:m]
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    pos, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=bits, positions=True,
                                        pairs=pairs)
    exp = expected(orc, kind, col, pr)
    np.testing.assert_array_equal(from_dev_u32(pos), exp)
    if pairs:
        erows, epos = orc.pairs_from_positions(exp)
        a = prs[: 2 * int(cnt.item())].cpu().numpy().view(np.uint32).reshape(-1, 2)
        a = a[np.argsort(a[:, 0], kind="stable")]
        np.testing.assert_array_equal(a[:, 0], erows)
        np.testing.assert_array_equal(a[:, 1], epos)


@pytest.mark.parametrize("bits", [1, 5, 8, 9, 11, 12])
def test_range_partition_with_a_larger_workspace(gj, cuda, bits):
    # one workspace, sized for the largest batch, for batches of every size below
    import torch

    for most, m in ((1_300_000, 1_200_000), (2_600_000, 2_489_000), (5_000_000, 4_950_000)):
        need = ctypes.c_size_t(0)
        assert gj.lib().gj_partition_workspace_size(most, bits, ctypes.byref(need)) == 0
        ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
        keys = torch.arange(m, device="cuda", dtype=torch.int64) * 7 % m
        rel = gj.range_partition(keys, 0, max(0, m.bit_length() - bits), bits, workspace=ws)
        assert torch.equal(keys[rel.rows.to(torch.int64)], rel.keys)
        assert torch.equal(torch.sort(rel.rows.to(torch.int64))[0], torch.arange(m, device="cuda"))


@pytest.mark.parametrize("prepared", [False, True])
@pytest.mark.parametrize("aligned", [False, True])
@pytest.mark.parametrize("kind,params", [("radix_spline", {}), ("btree", {"btree_node_keys": 8})])
def test_large_windows_of_positions(orc, gj, cuda, kind, params, aligned, prepared):
    # results in the relation's order (k_part_values): a column on and off the
    # sector boundary, the directory kept with the index or built for the call,
    # lower bounds and equal keys, a ragged last block
    import torch

    m = (1 << 22) + 4097
    rng = np.random.default_rng(3)
    col = column(rng, 300_006 if aligned else 300_007)
    pr = probes_for(rng, col, m)[:m]
    d_all = to_dev(torch, np.concatenate([np.zeros(4 if aligned else 1, dtype=np.uint64), col]))
    d_col = d_all[4:] if aligned else d_all[1:]
    assert (d_col.data_ptr() % 32 == 0) == aligned
    ix = gj.make_index(kind, **params).construct(None, d_col)
    if prepared:
        ix.prepare_partitioned()
    got, _, _ = ix.partitioned_inlj(to_dev(torch, pr))
    np.testing.assert_array_equal(from_dev_u32(got), expected(orc, kind, col, pr))


def test_large_windows_of_a_no_op_index(gj, cuda):
    # a window and a column large enough not to take the plain lookup
    import torch

    keys = gj.generate_sorted_keys((1 << 25) + 64, 0, 1 << 63, seed=3)
    probes = gj.generate_probes(keys, 3 << 24, theta=0.5, seed=4)
    got, _, _ = gj.make_index("no_op").construct(None, keys).partitioned_inlj(probes)
    assert bool((got == -1).all())
