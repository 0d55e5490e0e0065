"""Join materialisation, partitioned INLJ and the star-join aggregate on the
GPU against the CPU oracle."""
import ctypes

import numpy as np
import pytest

from test_lookup_gpu import column, expected, from_dev_u32, probes_for, to_dev

pytestmark = pytest.mark.gpu


def pairs_of(out_pairs, count):
    c = int(count.item())
    a = out_pairs[: 2 * c].cpu().numpy().view(np.uint32).reshape(-1, 2)
    return a[:, 0].copy(), a[:, 1].copy()


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("kind", ["binary_search", "btree", "harmonia", "radix_spline", "hash"])
@pytest.mark.parametrize("m", [0, 1, 31, 2047, 2048, 2049, 100003])
def test_inlj_pairs_match_oracle(orc, gj, cuda, kind, m, ordered):
    # in probe order, or (gj_inlj_pairs_unordered) the same set
    import torch

    rng = np.random.default_rng(m + 3)
    col = column(rng, 32 * 1000)
    pr = probes_for(rng, col, max(m, 1))[:m]
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    out, cnt = ix.inlj_pairs(to_dev(torch, pr) if m else torch.empty(0, dtype=torch.int64, device="cuda"),
                             ordered=ordered)
    rows, pos = pairs_of(out, cnt)
    if not ordered:
        order = np.argsort(rows, kind="stable")
        rows, pos = rows[order], pos[order]
    erows, epos = orc.pairs_from_positions(expected(orc, kind, col, pr))
    np.testing.assert_array_equal(rows, erows)
    np.testing.assert_array_equal(pos, epos)


@pytest.mark.parametrize("kind", ["btree", "learned", "no_op"])
@pytest.mark.parametrize("m", [4095, 4096, 4097, 3 * 1000 * 1000 + 17])
def test_inlj_pairs_compaction_tiles(orc, gj, cuda, kind, m):
    # plain pairs are positions first (parked in the upper half of the pairs
    # buffer), then an ordered compaction over 4096-probe tiles with a
    # look-back over many predecessors; the workspace is reused across calls
    import torch

    rng = np.random.default_rng(m)
    col = column(rng, 32 * 4000)
    pr = probes_for(rng, col, m)[:m]
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    d_pr = to_dev(torch, pr)
    ws = None
    for _ in range(2):
        out, cnt = ix.inlj_pairs(d_pr, workspace=ws)
        if ws is None:
            import ctypes

            need = ctypes.c_size_t(0)
            gj.lib().gj_inlj_pairs_workspace_size(m, ctypes.byref(need))
            ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
            out, cnt = ix.inlj_pairs(d_pr, workspace=ws)
        ix.inlj_pairs_status(ws, m)
        rows, pos = pairs_of(out, cnt)
        erows, epos = orc.pairs_from_positions(expected(orc, kind, col, pr))
        np.testing.assert_array_equal(rows, erows)
        np.testing.assert_array_equal(pos, epos)


def test_inlj_pairs_all_absent(orc, gj, cuda):
    import torch

    col = np.arange(0, 3200, dtype=np.uint64) * 2
    pr = np.arange(1, 6401, 2, dtype=np.uint64)  # odd keys: none present
    ix = gj.btree_index().construct(None, to_dev(torch, col))
    out, cnt = ix.inlj_pairs(to_dev(torch, pr))
    assert int(cnt.item()) == 0


@pytest.mark.parametrize("bits", [1, 4, 8, 12])
def test_range_partition_matches_oracle(orc, gj, cuda, bits):
    import torch

    rng = np.random.default_rng(bits)
    keys = rng.integers(0, 1 << 48, 300001, dtype=np.uint64)
    min_key, shift = 1 << 20, 48 - bits
    rel = gj.range_partition(to_dev(torch, keys), min_key, shift, bits)
    ok, orows, offs = orc.range_partition(keys, min_key, shift, bits)
    np.testing.assert_array_equal(rel.offsets.cpu().numpy().view(np.uint64), offs)
    gk = rel.keys.cpu().numpy().view(np.uint64)
    gr = rel.rows.cpu().numpy().view(np.uint32)
    np.testing.assert_array_equal(keys[gr], gk)
    # same tuples per partition (the order inside a partition is not fixed)
    for p in range(1 << bits):
        a, b = int(offs[p]), int(offs[p + 1])
        np.testing.assert_array_equal(np.sort(gr[a:b]), np.sort(orows[a:b]))


@pytest.mark.parametrize("kind", ["binary_search", "btree", "harmonia", "radix_spline"])
@pytest.mark.parametrize("window", [0, 1000, 65536])
def test_partitioned_inlj_equals_plain(orc, gj, cuda, kind, window):
    import torch

    rng = np.random.default_rng(window + 17)
    col = column(rng, 32 * 5000)
    pr = probes_for(rng, col, 120000)
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    pos, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=0, positions=True,
                                        pairs=True)
    exp = expected(orc, kind, col, pr)
    np.testing.assert_array_equal(from_dev_u32(pos), exp)
    rows, bpos = pairs_of(prs, cnt)
    erows, epos = orc.pairs_from_positions(exp)
    order = np.argsort(rows, kind="stable")
    np.testing.assert_array_equal(rows[order], erows)
    np.testing.assert_array_equal(bpos[order], epos)


@pytest.mark.parametrize("bits", [8, 10, 12])
def test_partitioned_inlj_fanouts(orc, gj, cuda, bits):
    import torch

    rng = np.random.default_rng(bits + 50)
    col = column(rng, 1 << 18)
    pr = probes_for(rng, col, 200000)
    ix = gj.btree_index().construct(None, to_dev(torch, col))
    pos, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), radix_bits=bits, pairs=True)
    exp = orc.exact_lookup(col, pr)
    np.testing.assert_array_equal(from_dev_u32(pos), exp)
    rows, bpos = pairs_of(prs, cnt)
    erows, epos = orc.pairs_from_positions(exp)
    order = np.argsort(rows, kind="stable")
    np.testing.assert_array_equal(rows[order], erows)
    np.testing.assert_array_equal(bpos[order], epos)


@pytest.mark.parametrize("kind", ["btree", "harmonia", "radix_spline", "binary_search", "learned", "hash"])
def test_partitioned_pairs_sorted_tiles(orc, gj, cuda, kind):
    # tiles of equal keys, a tile spanning the whole key range, many windows
    import torch

    rng = np.random.default_rng(99)
    col = column(rng, 32 * 20000)
    pr = np.concatenate([np.full(5000, col[777], dtype=np.uint64), probes_for(rng, col, 300000),
                         np.array([0, (1 << 64) - 1], dtype=np.uint64), np.full(3000, col[-1], dtype=np.uint64)])
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    exp = expected(orc, kind, col, pr)
    erows, epos = orc.pairs_from_positions(exp)
    for window, bits in ((len(pr), 8), (70001, 10), (4096, 12)):
        _, prs, cnt = ix.partitioned_inlj(to_dev(torch, pr), window_size=window, radix_bits=bits, positions=False,
                                          pairs=True)
        rows, bpos = pairs_of(prs, cnt)
        order = np.argsort(rows, kind="stable")
        np.testing.assert_array_equal(rows[order], erows, err_msg=f"{kind} window {window}")
        np.testing.assert_array_equal(bpos[order], epos, err_msg=f"{kind} window {window}")


def star_inputs(rng, nfact, ndim):
    dim = np.arange(1, ndim + 1, dtype=np.uint64)
    flag = np.zeros(ndim, dtype=np.uint8)
    flag[rng.choice(ndim, ndim // 6, replace=False)] = 1
    fk = rng.integers(1, ndim + 1, nfact).astype(np.uint32)
    fk[rng.integers(0, nfact, nfact // 50)] = ndim + 7  # dangling foreign keys
    date = rng.integers(0, 2556, nfact).astype(np.uint32)
    price = rng.integers(90000, 10500001, nfact).astype(np.int64)
    disc = rng.integers(0, 11, nfact).astype(np.int64)
    return dim, flag, fk, date, price, disc


@pytest.mark.parametrize("sorted_batches", [False, True])
@pytest.mark.parametrize("kind", ["btree", "harmonia", "binary_search", "radix_spline"])
@pytest.mark.parametrize("nfact", [0, 1, 4095, 4097, 600000])
def test_star_join_matches_oracle(orc, gj, cuda, kind, nfact, sorted_batches):
    import torch

    rng = np.random.default_rng(nfact + 1)
    ndim = 20000
    dim, flag, fk, date, price, disc = star_inputs(rng, max(nfact, 1), ndim)
    fk, date, price, disc = fk[:nfact], date[:nfact], price[:nfact], disc[:nfact]
    lo, hi = 1000, 1030
    ix = gj.make_index(kind).construct(None, to_dev(torch, dim))
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(dt).cuda()
    out = gj.star_join_sum(ix, t(fk.view(np.int32), torch.int32), t(date.view(np.int32), torch.int32),
                           t(price, torch.int64), t(disc, torch.int64), t(flag, torch.uint8), lo, hi,
                           sorted_batches=sorted_batches)
    num, den = orc.star_join(fk, date, price, disc, dim, flag, lo, hi)
    got = out.cpu().numpy()
    assert int(got[0]) == num and int(got[1]) == den


def test_star_join_full_window_and_empty_window(orc, gj, cuda):
    import torch

    rng = np.random.default_rng(99)
    dim, flag, fk, date, price, disc = star_inputs(rng, 100000, 5000)
    ix = gj.btree_index().construct(None, to_dev(torch, dim))
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a)).to(dt).cuda()
    args = (t(fk.view(np.int32), torch.int32), t(date.view(np.int32), torch.int32), t(price, torch.int64),
            t(disc, torch.int64), t(flag, torch.uint8))
    for lo, hi in ((0, 1 << 31), (500, 500), (2555, 2556), (100, 900)):
        num, den = orc.star_join(fk, date, price, disc, dim, flag, lo, hi)
        for sorted_batches in (False, True):  # every row passes / none / a few / a third
            got = gj.star_join_sum(ix, *args, lo, hi, sorted_batches=sorted_batches).cpu().numpy()
            assert (int(got[0]), int(got[1])) == (num, den), (lo, hi, sorted_batches)


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("kind", ["btree", "radix_spline", "learned"])
@pytest.mark.parametrize("m", [0, 1, 4097, 300001])
def test_inlj_pairs_host_buffers(orc, gj, cuda, kind, m, ordered):
    # probes, pairs and count in pinned host memory, read and written by the
    # kernels; unordered: the same set of pairs, tiles in the order they finish
    import torch

    rng = np.random.default_rng(m + 11)
    col = column(rng, 32 * 3000)
    pr = probes_for(rng, col, max(m, 1))[:m]
    ix = gj.make_index(kind).construct(None, to_dev(torch, col))
    h_pr = torch.from_numpy(pr.view(np.int64).copy()).pin_memory()
    h_pairs = torch.full((2 * max(m, 1),), -1, dtype=torch.int32).pin_memory()
    h_cnt = torch.full((1,), -1, dtype=torch.int64).pin_memory()
    ix.inlj_pairs_host(h_pr, h_pairs, h_cnt, ordered=ordered)
    torch.cuda.synchronize()
    c = int(h_cnt[0])
    got = h_pairs[: 2 * c].numpy().view(np.uint32).reshape(-1, 2)
    erows, epos = orc.pairs_from_positions(expected(orc, kind, col, pr))
    if not ordered:
        got = got[np.argsort(got[:, 0], kind="stable")]
    np.testing.assert_array_equal(got[:, 0], erows)
    np.testing.assert_array_equal(got[:, 1], epos)


@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("m", [(1 << 24) + 54321, 3 * (1 << 24) + 5])
def test_inlj_pairs_host_buffers_large(orc, gj, cuda, m, ordered):
    # tens of millions of probes from host buffers: every pair (in probe
    # order unless unordered), the status reads clean
    import torch

    rng = np.random.default_rng(3)
    col = column(rng, 1 << 16)
    pr = col[rng.integers(0, len(col), m)]
    pr[::7] = pr[::7] + np.uint64(1)  # some absent keys
    ix = gj.btree_index().construct(None, to_dev(torch, col))
    h_pr = torch.from_numpy(pr.view(np.int64).copy()).pin_memory()
    h_pairs = torch.full((2 * m,), -1, dtype=torch.int32).pin_memory()
    h_cnt = torch.full((1,), -1, dtype=torch.int64).pin_memory()
    need = ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(need))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    ix.inlj_pairs_host(h_pr, h_pairs, h_cnt, ws, ordered=ordered)
    torch.cuda.synchronize()
    ix.inlj_pairs_status(ws, m)
    c = int(h_cnt[0])
    got = h_pairs[: 2 * c].numpy().view(np.uint32).reshape(-1, 2)
    erows, epos = orc.pairs_from_positions(orc.exact_lookup(col, pr))
    if not ordered:
        got = got[np.argsort(got[:, 0], kind="stable")]
    np.testing.assert_array_equal(got[:, 0], erows)
    np.testing.assert_array_equal(got[:, 1], epos)


@pytest.mark.parametrize("m", [(1 << 22) + 12345, 3 * (1 << 22) + 7])
def test_inlj_pairs_large(orc, gj, cuda, m):
    # millions of probes through the two-pass pairs and the allocation-free
    # entry point: pairs in probe order, clean status
    import torch

    rng = np.random.default_rng(m % 1000)
    col = column(rng, 1 << 16)
    pr = col[rng.integers(0, len(col), m)]
    pr[::5] = pr[::5] + np.uint64(1)  # absent keys
    ix = gj.btree_index().construct(None, to_dev(torch, col))
    d_pr = to_dev(torch, pr)
    need = ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_workspace_size(m, ctypes.byref(need))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out, cnt = ix.inlj_pairs(d_pr, workspace=ws)
    ix.inlj_pairs_status(ws, m)
    rows, pos = pairs_of(out, cnt)
    erows, epos = orc.pairs_from_positions(orc.exact_lookup(col, pr))
    np.testing.assert_array_equal(rows, erows)
    np.testing.assert_array_equal(pos, epos)
    out2, cnt2 = ix.inlj_pairs_noalloc(d_pr, torch.empty_like(out), torch.zeros_like(cnt))
    rows2, pos2 = pairs_of(out2, cnt2)
    np.testing.assert_array_equal(rows2, erows)
    np.testing.assert_array_equal(pos2, epos)


@pytest.mark.parametrize("kind", ["btree", "binary_search", "harmonia", "radix_spline", "learned", "hash"])
@pytest.mark.parametrize("dist", ["DIST_UNIFORM", "DIST_LOGNORMAL"])
@pytest.mark.parametrize("m", [3 << 24, (3 << 24) + 4097])
def test_pairs_by_partition(gj, cuda, kind, dist, m):
    # calls large enough to partition their probes first: the same pairs, in
    # probe order, as the index's own lookups give, on the offered workspace
    # and on one that has no room for it
    import torch

    n = (1 << 25) + 64
    keys = gj.generate_sorted_keys(n, getattr(gj, dist), 1 << 63, seed=5)
    ix = gj.make_index(kind).construct(None, keys)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    probes[:4] = torch.tensor([0, 1, -1, -2], dtype=torch.int64, device="cuda")  # both ends of the key range
    pos = ix.lookup(probes)
    rows = torch.nonzero(pos != -1).flatten()
    small, offered = ctypes.c_size_t(0), ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(small))
    gj.lib().gj_inlj_pairs_workspace_size(m, ctypes.byref(offered))
    assert offered.value > 6 * m > small.value
    for nbytes in (offered.value, small.value):
        ws = torch.full((nbytes,), 0xA5, dtype=torch.uint8, device="cuda")
        pairs, count = ix.inlj_pairs(probes, workspace=ws)
        ix.inlj_pairs_status(ws, m)
        assert int(count) == rows.numel()
        got = pairs[: 2 * int(count)].view(-1, 2)
        assert torch.equal(got[:, 0].to(torch.int64), rows)
        assert torch.equal(got[:, 1], pos[rows])


@pytest.mark.parametrize("kind", ["btree", "binary_search", "hash"])
@pytest.mark.parametrize("column", ["clusters", "dense", "end_of_range"])
def test_pairs_by_partition_start_tables(gj, cuda, kind, column):
    # columns for which the partitioned pairs' table stays the lookups' own
    # (clusters), has two keys a bucket (dense) or ends at the largest key with
    # nearly all keys in its first buckets (end_of_range)
    import torch

    m = (1 << 25) + 257
    if column == "clusters":
        keys = gj.generate_sorted_keys(1 << 26, gj.DIST_CLUSTERS, 1 << 63, seed=5)
    else:
        keys = torch.arange((1 << 25) + 64, dtype=torch.int64, device="cuda") + 7
        if column == "end_of_range":
            keys[-1] = -1  # 2^64 - 1
    ix = gj.make_index(kind).construct(None, keys)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1 if column == "clusters" else 0.0, seed=6)
    probes[:6] = torch.tensor([0, 6, 7, -1, -2, (1 << 25) + 71], dtype=torch.int64, device="cuda")
    pos = ix.lookup(probes)
    rows = torch.nonzero(pos != -1).flatten()
    pairs, count = ix.inlj_pairs(probes)
    assert int(count) == rows.numel()
    got = pairs[: 2 * int(count)].view(-1, 2)
    assert torch.equal(got[:, 0].to(torch.int64), rows)
    assert torch.equal(got[:, 1], pos[rows])


@pytest.mark.parametrize("kind,n", [("hash", 1 << 25), ("btree", 1 << 20), ("btree", 20_000_000)])
def test_pairs_workspace_without_a_partition(gj, cuda, kind, n):
    # an index whose pairs are never partitioned: large calls take no room for it
    import torch

    m = (1 << 25) + 3
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    ix = gj.make_index(kind).construct(None, keys)
    least, need = ctypes.c_size_t(0), ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(least))
    assert gj.lib().gj_index_inlj_pairs_workspace_size(ix.handle, m, ctypes.byref(need)) == 0
    assert need.value == least.value
    probes = gj.generate_probes(keys, m, theta=0.5, seed=6)
    out, count = torch.empty(2 * m, dtype=torch.int32, device="cuda"), torch.empty(1, dtype=torch.int64, device="cuda")
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    ix.inlj_pairs(probes, out, count)
    assert torch.cuda.max_memory_allocated() - before < least.value + (4 << 20)
    assert int(count) == m


def test_pairs_with_little_memory(gj, cuda, monkeypatch):
    # no memory for the room to partition: the pairs come without it
    import torch

    n, m = (1 << 25) + 64, (1 << 25) + 3
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    ix = gj.btree_index().construct(None, keys)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    pairs, count = ix.inlj_pairs(probes)
    sizes, real = [], gj._workspace

    def scarce(nbytes, device):
        sizes.append(nbytes)
        if nbytes > m:
            raise torch.cuda.OutOfMemoryError("full")
        return real(nbytes, device)

    monkeypatch.setattr(gj, "_workspace", scarce)
    again, recount = ix.inlj_pairs(probes)
    assert len(sizes) == 2 and sizes[0] > 6 * m > sizes[1]
    assert int(count) == int(recount) and torch.equal(pairs[: 2 * int(count)], again[: 2 * int(count)])


def test_partition_scratch_is_aligned(gj, cuda):
    # the partition's arrays behind the state of an ordered call start on a
    # 256-byte boundary of the workspace, as the state itself does
    import torch

    n, m = (1 << 25) + 64, (1 << 25) + 257
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    ix = gj.btree_index().construct(None, keys)
    probes = gj.generate_probes(keys, m, theta=0.5, seed=6)
    least, need = ctypes.c_size_t(0), ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(least))
    gj.lib().gj_index_inlj_pairs_workspace_size(ix.handle, m, ctypes.byref(need))
    ws = torch.full((need.value,), 0xA5, dtype=torch.uint8, device="cuda")
    _, count = ix.inlj_pairs(probes, workspace=ws)
    assert int(count) == m and ws.data_ptr() % 256 == 0
    first = int(torch.nonzero(ws[least.value: least.value + 4096] != 0xA5)[0])
    assert (least.value + first) % 256 == 0


def route_of(gj, ix, probes):
    """(pairs, count, how) of an ordered call on the workspace its index asks
    for: "plain" (no room to partition is asked for, or none is touched),
    "stayed" (it was sampled, and its probes were searched as they came) or
    "partitioned" (the partition's tables, first in that room, were written)"""
    import torch

    m = probes.numel()
    least, need = ctypes.c_size_t(0), ctypes.c_size_t(0)
    gj.lib().gj_inlj_pairs_host_workspace_size(m, ctypes.byref(least))
    gj.lib().gj_index_inlj_pairs_workspace_size(ix.handle, m, ctypes.byref(need))
    ws = torch.full((need.value,), 0xA5, dtype=torch.uint8, device="cuda")
    pairs, count = ix.inlj_pairs(probes, workspace=ws)
    ix.inlj_pairs_status(ws, m)
    room = ws[least.value:]
    if not bool((room != 0xA5).any()):
        return pairs, count, "plain"
    return pairs, count, "partitioned" if bool((room[256:4096] != 0xA5).any()) else "stayed"


def skew(torch, gj, keys, m, form):
    if form == "even":
        return gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    if form == "skewed":
        return gj.generate_probes(keys, m, theta=1.5, absent_fraction=0.1, seed=6)
    p = gj.generate_probes(keys, m, theta=0.0, seed=6)
    p = torch.sort(p)[0] if int(keys[-1]) >= 0 else p
    if form == "nearly sorted":  # shuffled inside windows of 4096
        q = p[: m // 4096 * 4096].view(-1, 4096)
        p[: m // 4096 * 4096] = q[:, torch.randperm(4096, device="cuda")].reshape(-1)
    return p


@pytest.mark.parametrize("column", ["uniform", "lognormal", "clusters", "whole range"])
@pytest.mark.parametrize("form", ["even", "skewed", "sorted", "nearly sorted"])
@pytest.mark.parametrize("kind", ["btree", "binary_search"])
def test_ordered_pairs_look_at_their_probes(orc, gj, cuda, kind, form, column):
    # even probes are partitioned; skewed ones and those in order or nearly so
    # are searched as they come -- the same pairs in the same order, against the
    # oracle, over a finer and a coarse table (clusters) and up to 2^64 - 1
    import torch

    m = (1 << 25) + 257
    n = (1 << 26) if column == "clusters" else (1 << 25) + 64
    if column == "whole range":
        if form in ("sorted", "nearly sorted"):
            pytest.skip("probes are sorted as signed numbers")
        keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5) * 2  # above 2^63 too
        keys[0], keys[-1] = 0, -1  # 2^64 - 1
    else:
        keys = gj.generate_sorted_keys(n, getattr(gj, "DIST_" + column.upper()), 1 << 63, seed=5)
    probes = skew(torch, gj, keys, m, form)
    probes[:4] = torch.tensor([0, 1, -1, -2], dtype=torch.int64, device="cuda")
    ix = gj.make_index(kind).construct(None, keys)
    pairs, count, how = route_of(gj, ix, probes)
    assert how == ("partitioned" if form == "even" else "stayed")
    col, pr = keys.cpu().numpy().view(np.uint64), probes.cpu().numpy().view(np.uint64)
    exp = (orc.exact_lookup if kind == "btree" else orc.bs_lookup)(col, pr)
    rows, pos = orc.pairs_from_positions(exp)
    got = pairs[: 2 * int(count)].cpu().numpy().view(np.uint32).reshape(-1, 2)
    assert int(count) == len(rows)
    np.testing.assert_array_equal(got[:, 0], rows)
    np.testing.assert_array_equal(got[:, 1], pos)


@pytest.mark.parametrize("kind,n,m,how", [("hash", 1 << 25, (1 << 25) + 5, "plain"),
                                          ("btree", 20_000_000, (1 << 25) + 5, "plain"),
                                          ("btree", 3 << 23, (1 << 25) + 5, "plain"),
                                          ("btree", (3 << 23) + 64, (1 << 25) + 5, "partitioned"),
                                          ("btree", (3 << 23) + 64, 1 << 25, "partitioned"),
                                          ("btree", (3 << 23) + 64, (1 << 25) - 1, "plain"),
                                          ("radix_spline", (3 << 22) + 64, (1 << 25) + 5, "partitioned"),
                                          ("learned", (3 << 22) + 64, (1 << 25) + 5, "partitioned")])
def test_which_ordered_pairs_are_partitioned(gj, cuda, kind, n, m, how):
    import torch

    kw = {"learned_steps": 20} if kind == "learned" else {}
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    ix = gj.make_index(kind, **kw).construct(None, keys)
    probes = gj.generate_probes(keys, m, theta=0.5, absent_fraction=0.1, seed=6)
    pairs, count, taken = route_of(gj, ix, probes)
    assert taken == how
    pos = ix.lookup(probes)
    rows = torch.nonzero(pos != -1).flatten()
    got = pairs[: 2 * int(count)].view(-1, 2)
    assert torch.equal(got[:, 0].to(torch.int64), rows) and torch.equal(got[:, 1], pos[rows])


def test_partitioned_pairs_under_capture(gj, cuda):
    # one captured call, replayed on probes that are partitioned and on probes
    # that are not: the choice is made on the device
    import torch

    n, m = (1 << 25) + 64, (1 << 25) + 257
    keys = gj.generate_sorted_keys(n, gj.DIST_UNIFORM, 1 << 63, seed=5)
    ix = gj.btree_index().construct(None, keys)
    probes = skew(torch, gj, keys, m, "even")
    need = ctypes.c_size_t(0)
    gj.lib().gj_index_inlj_pairs_workspace_size(ix.handle, m, ctypes.byref(need))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    pairs, count = torch.empty(2 * m, dtype=torch.int32, device="cuda"), torch.empty(1, dtype=torch.int64, device="cuda")
    ix.inlj_pairs(probes, pairs, count, ws)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ix.inlj_pairs(probes, pairs, count, ws)
    for form in ("skewed", "even", "sorted"):
        probes.copy_(skew(torch, gj, keys, m, form))
        graph.replay()
        pos = ix.lookup(probes)
        rows = torch.nonzero(pos != -1).flatten()
        assert int(count) == rows.numel()
        got = pairs[: 2 * int(count)].view(-1, 2)
        assert torch.equal(got[:, 0].to(torch.int64), rows) and torch.equal(got[:, 1], pos[rows])
