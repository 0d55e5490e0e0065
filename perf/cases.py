"""The probe path's workloads, as a program that uses gpujoin_gb300 runs them.

Each case is one call (or one short sequence of calls) through the package's
public entry points, with default arguments wherever a user would leave them:

  lookup     positions of a probe column, one index of any kind
  pairs      (probe row, build position) pairs in probe order; with absent
             keys the caller reads the count and marks the rest unused
  partition  range_partition with the reference's fixed fanout (2^11), then
             partitioned_lookup of the relation into a positions column
  windowed   partitioned_inlj of an index prepared for it, positions out
  host       pairs from pinned host probes into pinned host buffers
  star       the Q14-shaped star join: date filter, dimension probe, sums
  batch      a planned stream of batches against several indexes, replayed
             through the plan's graph

Outputs are whole numbers (positions, rows, counts, sums), so they have one
right value each; there is nothing to compare in 64 bits.
"""
import math

import numpy as np
import torch

import gpujoin_gb300 as gj

UPPER = 1 << 63


def listed():
    return [
        # a point query's worth of keys against the reference's default table
        # (10^6 rows): the smallest call, all launch and latency
        {"name": "lookup_1k", "op": "lookup", "kind": "btree", "n": 1_000_000, "m": 1_000, "dist": "uniform",
         "theta": 0.0, "absent": 0.0},
        # experiment_config's defaults: 10^8 Zipf(1.25) lookups into 10^6 rows
        {"name": "lookup_default", "op": "lookup", "kind": "btree", "n": 1_000_000, "m": 100_000_000,
         "dist": "uniform", "theta": 1.25, "absent": 0.0},
        # the headline benchmark: foreign-key join of 2^28 Zipf(0.5) probes
        # with a 2^26-key B+tree, pairs in probe order
        {"name": "pairs_headline", "op": "pairs", "kind": "btree", "n": 1 << 26, "m": 1 << 28, "dist": "uniform",
         "theta": 0.5, "absent": 0.0},
        # hash join of odd-sized tables, one probe in ten without a partner
        {"name": "pairs_hash", "op": "pairs", "kind": "hash", "n": 20_000_003, "m": 50_000_017, "dist": "uniform",
         "theta": 0.0, "absent": 0.1},
        # the learned index on the skewed column it is made for, some keys absent
        {"name": "learned_lognormal", "op": "lookup", "kind": "learned", "n": 1 << 27, "m": 1 << 26,
         "dist": "lognormal", "theta": 0.0, "absent": 0.05},
        # the plain index the others are held against
        {"name": "binary_search", "op": "lookup", "kind": "binary_search", "n": 1 << 26, "m": 1 << 26,
         "dist": "uniform", "theta": 0.5, "absent": 0.0},
        # the reference's second tree, clustered keys (ids handed out in runs)
        {"name": "harmonia_clusters", "op": "lookup", "kind": "harmonia", "n": 1 << 26, "m": 1 << 26,
         "dist": "clusters", "theta": 0.5, "absent": 0.0},
        # partition first, look up after: the reference's two operators by hand
        {"name": "partition_lookup", "op": "partition", "kind": "radix_spline", "n": 1 << 26, "m": 1 << 27,
         "dist": "uniform", "theta": 0.5, "absent": 0.0, "radix_bits": 11},
        # the partitioned join of the largest benchmark configuration
        {"name": "windowed_large", "op": "windowed", "kind": "btree", "n": 1 << 28, "m": 1 << 29, "dist": "uniform",
         "theta": 0.5, "absent": 0.0, "radix_bits": 0},
        # probes and pairs in pinned host memory, an odd count of them
        {"name": "host_pairs", "op": "host", "kind": "btree", "n": 1 << 26, "m": 33_333_333, "dist": "uniform",
         "theta": 0.5, "absent": 0.0},
        # TPC-H Q14 at scale factor 1: 6M lineitems, 200k parts, one month
        {"name": "star_sf1", "op": "star", "kind": "btree", "facts": 6_000_000, "dims": 200_000, "days": 30},
        # a serving tick: batches of uneven size against eight indexes
        {"name": "batch_stream", "op": "batch", "n": 1 << 24, "batches": 512, "median": 65_536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["lookup", "lookup", "pairs", "partition", "windowed", "host", "star", "batch"])
    if op == "star":
        return {"op": op, "kind": rng.choice(["btree", "harmonia"]), "facts": _log_int(rng, 100_000, 60_000_000),
                "dims": 32 * _log_int(rng, 300, 60_000), "days": _log_int(rng, 7, 365)}
    if op == "batch":
        return {"op": op, "n": _log_int(rng, 1 << 18, 1 << 24), "batches": _log_int(rng, 8, 512),
                "median": _log_int(rng, 1_000, 65_536)}
    kind = rng.choice(["btree", "harmonia", "binary_search", "radix_spline", "learned", "hash"])
    n = _log_int(rng, 1_000, 1 << 26)
    case = {"op": op, "kind": kind, "n": n, "m": _log_int(rng, 1_000, 1 << 26),
            "dist": rng.choice(["uniform", "uniform", "lognormal", "clusters"]),
            "theta": rng.choice([0.0, 0.5, 0.8, 1.25]), "absent": rng.choice([0.0, 0.0, 0.05, 0.1])}
    if kind == "harmonia":
        case["n"] = -(-n // 32) * 32  # its columns hold whole nodes
    if op == "partition":
        case["radix_bits"] = rng.choice([8, 11])
    if op == "windowed":
        case["m"] = _log_int(rng, 1_000_000, 1 << 28)
        case["radix_bits"] = rng.choice([0, 0, 8])
    if op == "host":
        case["m"] = _log_int(rng, 1_000, 33_333_333)
    return case


_DIST = {"uniform": gj.DIST_UNIFORM, "lognormal": gj.DIST_LOGNORMAL, "clusters": gj.DIST_CLUSTERS}


def _star(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nf, nd = case["facts"], case["dims"]

    def column(lo, hi, dtype):
        return torch.randint(lo, hi, (nf,), generator=g, dtype=dtype, device="cuda")

    flag = (torch.randint(0, 6, (nd,), generator=g, device="cuda") == 0).to(torch.uint8)
    parts = torch.arange(1, nd + 1, dtype=torch.int64, device="cuda")
    return {"op": "star", "index": gj.make_index(case["kind"]).construct(None, parts), "flag": flag,
            "fk": column(1, nd + 1, torch.int32), "date": column(0, 2556, torch.int32),
            "price": column(90_000, 10_500_001, torch.int64), "disc": column(0, 11, torch.int64),
            "lo": 1000, "hi": 1000 + case["days"]}


# kinds, sizes (halvings of the largest) and distributions of a stream's indexes
_STREAM = [("btree", 0, "uniform"), ("harmonia", 1, "uniform"), ("radix_spline", 2, "lognormal"),
           ("learned", 0, "lognormal"), ("btree", 3, "lognormal"), ("harmonia", 4, "uniform"),
           ("hash", 2, "uniform"), ("binary_search", 4, "uniform")]


def _batch(case, seed):
    columns, indexes = [], []
    for i, (kind, halvings, dist) in enumerate(_STREAM):
        n = -(-(case["n"] >> halvings) // 32) * 32
        columns.append(gj.generate_sorted_keys(n, _DIST[dist], UPPER, seed=seed * 16 + i))
        indexes.append(gj.make_index(kind).construct(None, columns[-1]))
    nb = case["batches"]
    rng = np.random.default_rng(nb)  # the tick's shape is the case's, its keys the seed's
    sizes = np.exp(rng.normal(math.log(case["median"]), 1.6, nb)).clip(100, 4 << 20).astype(np.int64)
    which = rng.integers(0, len(indexes), nb).astype(np.uint32)
    offsets = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    probes = torch.empty(int(sizes.sum()), dtype=torch.int64, device="cuda")
    for b in range(nb):
        probes[int(offsets[b]): int(offsets[b] + sizes[b])] = gj.generate_probes(
            columns[which[b]], int(sizes[b]), theta=0.8, seed=seed * 4096 + b)
    return {"op": "batch", "plan": gj.batch_plan(indexes, which, offsets.astype(np.uint64), sizes.astype(np.uint64)),
            "probes": probes, "out": torch.empty(probes.numel(), dtype=torch.int32, device="cuda")}


def prepare(case, seed):
    op = case["op"]
    if op == "star":
        return _star(case, seed)
    if op == "batch":
        return _batch(case, seed)
    keys = gj.generate_sorted_keys(case["n"], _DIST[case["dist"]], UPPER, seed=seed * 2 + 1)
    index = gj.make_index(case["kind"]).construct(None, keys)
    probes = gj.generate_probes(keys, case["m"], theta=case["theta"], absent_fraction=case["absent"], seed=seed * 2 + 2)
    state = {"op": op, "index": index, "probes": probes, "all_match": case["absent"] == 0.0}
    if op == "partition":
        low, high = int(keys[0]), int(keys[-1])
        used = (high - low).bit_length()
        state.update(low=low, shift=max(0, used - case["radix_bits"]), radix_bits=case["radix_bits"],
                     out=torch.empty(case["m"], dtype=torch.int32, device="cuda"))
    elif op == "windowed":
        index.prepare_partitioned()
        state.update(radix_bits=case["radix_bits"])
    elif op == "host":
        m = case["m"]
        state["probes"] = torch.empty(m, dtype=torch.int64, pin_memory=True).copy_(probes)
        state.update(pairs=torch.zeros(2 * m, dtype=torch.int32, pin_memory=True),
                     count=torch.zeros(1, dtype=torch.int64, pin_memory=True))
    return state


def run(state):
    op = state["op"]
    if op == "lookup":
        return state["index"].lookup(state["probes"])
    if op == "pairs":
        pairs, count = state["index"].inlj_pairs(state["probes"])
        if not state["all_match"]:  # a join that may lose rows: the caller reads how many pairs there are
            pairs[2 * int(count):].fill_(-1)
        return pairs, count
    if op == "partition":
        rel = gj.range_partition(state["probes"], state["low"], state["shift"], state["radix_bits"])
        state["index"].partitioned_lookup(rel.keys, rel.rows, state["out"])
        return rel.offsets, state["out"]
    if op == "windowed":
        positions, _, _ = state["index"].partitioned_inlj(state["probes"], radix_bits=state["radix_bits"])
        return positions
    if op == "host":
        pairs, count = state["index"].inlj_pairs_host(state["probes"], state["pairs"], state["count"])
        if not state["all_match"]:
            torch.cuda.current_stream().synchronize()  # the count is the caller's to read from here on
            pairs[2 * int(count):].fill_(-1)
        return pairs, count
    if op == "star":
        return gj.star_join_sum(state["index"], state["fk"], state["date"], state["price"], state["disc"],
                                state["flag"], state["lo"], state["hi"])
    return state["plan"].run_graph(state["probes"], state["out"])


def work(case):
    """Bytes of one pass: every probe and result once, and the part of the key
    column the probes can touch (all of it, or a 32-byte sector each)."""
    if case["op"] == "star":
        passing = case["facts"] * case["days"] / 2556.0
        return {"bytes": 4.0 * case["facts"] + passing * 20.0 + 9.0 * case["dims"], "flops": 0.0}
    if case["op"] == "batch":
        probes = case["batches"] * case["median"] * math.exp(1.6 * 1.6 / 2)
        keys = sum(case["n"] >> h for _, h, _ in _STREAM)
        return {"bytes": 12.0 * probes + min(8.0 * keys, 32.0 * probes), "flops": 0.0}
    n, m = case["n"], case["m"]
    result = 8.0 if case["op"] in ("pairs", "host") else 4.0
    return {"bytes": (8.0 + result) * m + min(8.0 * n, 32.0 * m), "flops": 0.0}
