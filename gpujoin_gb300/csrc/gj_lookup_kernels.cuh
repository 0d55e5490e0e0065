// gj_lookup_kernels.cuh -- the probe kernels and their launchers, shared by
// the translation units that instantiate them: each index kind (and B+tree
// node width) is compiled in one unit (gj_lookup*.cu), so the units build in
// parallel.  Everything but the call interface has internal linkage.
//
// Replaces lookup_kernel (src/index_lookup_common.cuh:217-245),
// partitioned_lookup_kernel (src/index_lookup_partitioning.cu:218-248) and
// ij_lookup_kernel (src/tpch/tpch_14_ij.cu:371-407).
//
// Lookups of scattered probes start at an entry of a start table (key start
// table, B+tree or Harmonia node table) and stage nothing; the sampled keys
// of a binary search without a table, and the top B+tree levels that the
// sorted-tile kernels descend once a tile, are staged in shared memory once
// per block.  Probe keys are streamed with evict-first loads, results with
// streaming stores.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>
#include <utility>

#include "gj_internal.h"

namespace gj {

// one launch of a probe kernel for an index, as passed between the units
enum class lookup_action { positions, scatter, pairs, sorted_pairs, sorted_positions };
struct lookup_call {
    lookup_action action;
    const uint64_t* keys;  // probes, or the keys of a partitioned relation
    const uint32_t* rows;  // row ids of a partitioned relation (scatter), else null
    uint64_t m;
    uint32_t* out;         // positions (positions, scatter) or pairs
    uint64_t* d_count;
    void* ws;
    size_t ws_bytes;
    uint32_t* stash;       // pairs: room for m positions (for two passes), or null (host buffers)
    cudaStream_t s;
    // test hook of the bounded waits (gj_debug_inlj_pairs_stalled): a spin
    // limit other than kSpinLimit (0 = default) and a first tile left
    // unclaimed, so that every look-back runs out
    uint32_t spin_limit;
    bool skip_first_tile;
    // pairs (single pass): tiles placed by one atomicAdd each instead of in
    // probe order
    bool unordered;
};

// per-kind entry points, each defined in one unit
int lookup_call_bs(const gj_index* idx, const lookup_call& c);
int lookup_call_noop(const gj_index* idx, const lookup_call& c);
int lookup_call_harmonia(const gj_index* idx, const lookup_call& c);
int lookup_call_rs(const gj_index* idx, const lookup_call& c);
int lookup_call_learned(const gj_index* idx, const lookup_call& c);
int lookup_call_hash(const gj_index* idx, const lookup_call& c);
template <int W>
int lookup_call_btree(const gj_index* idx, const lookup_call& c);  // the widths of btree_dispatch:
template <> int lookup_call_btree<4>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<7>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<8>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<15>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<16>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<32>(const gj_index* idx, const lookup_call& c);
template <> int lookup_call_btree<64>(const gj_index* idx, const lookup_call& c);

namespace {


constexpr int kBlock = 256;
// Resident blocks per SM each lookup kernel is compiled for: the register
// cap.  A search is a chain of dependent loads and the warps of an SM are
// what keeps loads in flight, so the tree and search kinds are capped at 32
// registers (8 blocks of 256 threads, full occupancy), which they meet
// without spilling; the learned index keeps 64 for its MLP root.
// GJ_MIN_BLOCKS overrides every kind (tuning builds).
#ifdef GJ_MIN_BLOCKS
#define GJ_BLOCKS(n) GJ_MIN_BLOCKS
#else
#define GJ_BLOCKS(n) (n)
#endif

// ---------------------------------------------------------------------------
// per-index lookup functors
// ---------------------------------------------------------------------------
struct stage_desc {
    const uint64_t* src0;
    const uint64_t* src1;
    uint32_t words0;
    uint32_t words1;
};

// Each op searches one probe.  lookup<kScattered> picks the L2 classes:
// scattered probes (operator()) keep the inner levels and stream the
// column; the partitioned kernels, whose nearby probes reuse column sectors
// and touch a slice of the tree, use the default class.
struct op_bs {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 8;
    static constexpr bool kStaged = true;
    bs_view v;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t* cache, uint64_t key) const {
        return bs_lookup(v, cache, key);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
// lookups through the index's key start table: the lower bound (binary
// search) or the position of an equal key (the default B+tree over a column
// small enough for the table to replace its levels)
template <bool kExact>
struct op_start {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 4;
    static constexpr bool kStaged = false;
    key_start t;
    const uint64_t* col;
    uint32_t n;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t key) const {
        bool eq;
        const uint32_t lb = start_lower_bound<kScattered>(t, col, n, key, &eq);
        return (kExact ? eq : lb < n) ? lb : kInvalid;
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
// Trees: a scattered lookup starts at its bucket's entry of the start table,
// over large columns nearly always below the levels that fit shared memory, so
// there only the sorted tiles (whose common node is searched from the root)
// stage them; the kernels without them keep the room for L1 and have nothing to
// load before the first probe.  kSm (plain nodes over up to kStageKeys keys):
// blocks of several probes a thread stage them, as all or most levels of such a
// tree lie there (6 M probes through nodes of 8 keys: 4096 keys 90 us, 118
// unstaged, 2^16 keys of Zipf(1.25) 116 / 137, uniform 131 / 133; from 2^20 on the
// room is worth more to L1, 34 M unordered pairs through nodes of 4 keys over 2^22
// keys 984 / 676);
// those of one probe a thread would pay for it at every block and do not.
//
// Sorted tiles: an op with a tile_hint searches once per tile for what all
// keys of the tile's range share (for the B+tree: the deepest node on every
// path) and starts each probe's search there.
template <int W, bool kSm = false>
struct op_btree {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 8;
    static constexpr bool kStaged = kSm;
    btree_view v;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t* cache, uint64_t key) const {
        return btree_lookup<W, kScattered, kSm>(v, cache, key);
    }
    op_btree unstaged() const {
        op_btree o = *this;
        o.v.cached_levels = 0;
        return o;
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
    using tile_hint = btree_cursor;
    __device__ __forceinline__ tile_hint tile(const uint64_t* cache, uint64_t lo, uint64_t hi) const {
        return btree_common_node<W, false>(v, cache, lo, hi);
    }
    __device__ __forceinline__ uint32_t lookup_in_tile(const uint64_t* cache, uint64_t key, const tile_hint& h) const {
        return btree_lookup_from<W, false>(v, cache, key, h);
    }
};

template <class Op>
struct is_tree_nodes : std::false_type {};
template <int W, bool kSm>
struct is_tree_nodes<op_btree<W, kSm>> : std::true_type {};
constexpr uint64_t kStageKeys = 1ull << 18;

struct no_tile_hint {};
template <class Op, class = void>
struct tile_hint_of {
    using type = no_tile_hint;
};
template <class Op>
struct tile_hint_of<Op, std::void_t<typename Op::tile_hint>> {
    using type = typename Op::tile_hint;
};
struct op_harmonia {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 4;
    static constexpr bool kStaged = false;
    harmonia_view v;
    harmonia_child_base base;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t* cache, uint64_t key) const {
        return harmonia_lookup<kScattered, false>(v, cache, key, &base);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
struct op_rs {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 1;
    static constexpr bool kStaged = false;
    rs_view v;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t key) const {
        return rs_lookup<kScattered>(v, key);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
struct op_hash {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 8;
    static constexpr bool kStaged = false;
    hash_view v;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t key) const {
        return hash_lookup(v, key);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
struct op_noop {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 8;
    static constexpr bool kStaged = false;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t) const { return kInvalid; }
    __device__ __forceinline__ uint32_t operator()(const uint64_t*, uint64_t) const { return kInvalid; }
};
// the root parameters travel inside the op (a kernel argument): the MLP's
// FMAs read their weights from the constant bank
struct op_learned {
    static constexpr int kMinBlocks = GJ_BLOCKS(4);
    static constexpr int kLong = 8;
    static constexpr bool kStaged = false;
    learned_view v;
    learned_root_params p;
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t key) const {
        return learned_lookup<kScattered>(v, p.w, key);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};
// linear and segment-table roots: no network to evaluate, twice the warps
struct op_learned_plain {
    static constexpr int kMinBlocks = GJ_BLOCKS(8);
    static constexpr int kLong = 4;
    static constexpr bool kStaged = false;
    learned_view v;
    float p[2];
    template <bool kScattered = true>
    __device__ __forceinline__ uint32_t lookup(const uint64_t*, uint64_t key) const {
        return learned_lookup<kScattered, false>(v, p, key);
    }
    __device__ __forceinline__ uint32_t operator()(const uint64_t* cache, uint64_t key) const { return lookup(cache, key); }
};

__device__ __forceinline__ void stage_cache(uint64_t* dst, const stage_desc& sd) {
    for (uint32_t i = threadIdx.x; i < sd.words0; i += blockDim.x) dst[i] = __ldg(reinterpret_cast<const unsigned long long*>(sd.src0) + i);
    for (uint32_t i = threadIdx.x; i < sd.words1; i += blockDim.x)
        dst[sd.words0 + i] = __ldg(reinterpret_cast<const unsigned long long*>(sd.src1) + i);
    __syncthreads();
}

// ---------------------------------------------------------------------------
// plain lookup: out[i] = lookup(probes[i])
// ---------------------------------------------------------------------------
// One block per tile of kIt * kBlock probes (item k of thread t is
// probe tile + k * kBlock + t: coalesced).  The grid is not persistent: the
// hardware hands tiles to SMs as they free up, which balances SMs that run
// at different speeds (near and far HBM of the two dies) without a counter.
// A thread searches its probes one after another (a search is a chain of
// dependent loads; occupancy, not per-thread interleaving, keeps many loads
// in flight) and loads the next probe key before it searches the current
// one.  No per-thread arrays: the search runs with few live registers.


// Whether a lookup launch gives its threads Op::kLong probes each, one after
// another, or one.  One fills the chip from the fewest probes (65,536 probes
// into 2^26 keys: 84 us in 2048-probe blocks, 10 in 256-probe blocks) and
// keeps most loads in flight when the column's sectors come from DRAM (2^26
// probes into 2^26 keys 1568 against 1654 us); several save a block's start
// where the searches run from L2 (hash table of 2^20 keys 406 against 485 us
// with 8, key start table 534 against 569 with 4; RadixSpline is level).  Plain lookups take several up to 2^24 keys,
// where most sectors still hit L2 (24 M probes with 1 / 4: B+tree, uniform
// probes 358 / 352 us, Zipf(1.25) 212 / 189), and into a hash table, whose
// search is one load, at any size (2^26 keys with 1 / 4 / 8: uniform 548 / 559
// / 567, Zipf(1.25), which L1 and L2 serve, 160 / 133 / 132).  So do MLP roots,
// which are bound by issue (34 M probes into 20 M keys, 16 wide, 1294 / 1040).
constexpr uint64_t kL2Keys = 1ull << 23;  // columns of up to 64 MB stay in L2
template <class Op>
constexpr uint64_t kLookupLongKeys =
    std::is_same<Op, op_hash>::value || std::is_same<Op, op_learned>::value ? UINT64_MAX : 1ull << 24;
// The default B+tree's nodes are searched so a little further, in calls of 2^24
// probes and more (67 M probes with 1 / 8: 20 M uniform keys 1186 / 1116 us,
// lognormal 1254 / 1185; 2^25 keys, Zipf(0.8), 1224 / 1256), and its ordered
// pairs of that size take two passes, whose lookup can (1334 / 1261).  Scattered
// results bind the partitioned lookups of 2^25 probes and more, whose stores
// come from fewer warps at a time then (67 M into 20 M keys 2205 / 2089 us, 34 M
// through a RadixSpline of 2^25 keys with 1 / 4 910 / 807; 17 M probes, whose
// results fit L2, into 2^26 keys 385 / 513).
constexpr uint64_t kNodeLongKeys = 3ull << 23, kNodeLongProbes = 1ull << 24, kScatterLongProbes = 1ull << 25;
template <class Op>
constexpr bool kNodeSearch = is_tree_nodes<Op>::value;
template <class Op>
bool nodes_long(uint64_t n, uint64_t m) {
    return kNodeSearch<Op> && n <= kNodeLongKeys && m >= kNodeLongProbes;
}
// their ordered pairs up to 2^24 keys take the two passes as soon as the lookup
// does (6 M pairs, nodes of 15 keys over leaves of 8, 2^20 clustered keys, Zipf(1.25):
// 878 us in one pass, 702 in two; nodes of 8 over 4096 keys 163 / 110)
template <class Op>
bool nodes_two_passes(uint64_t n, uint64_t m, int sm_count) {
    return nodes_long<Op>(n, m) ||
           (kNodeSearch<Op> && n <= (1ull << 24) && m >= 16ull * sm_count * 8 * kBlock);
}
inline int long_blocks(uint64_t n, uint64_t m, bool* yes, uint64_t keys = kL2Keys) {
    device_info di;
    GJ_TRY(current_device_info(&di));
    *yes = n <= keys && m >= 16ull * di.sm_count * 8 * kBlock;  // 16 waves of a full chip
    return GJ_OK;
}

__device__ __forceinline__ uint64_t load_probe(const uint64_t* p, uint64_t i, uint64_t m) {
    return i < m ? __ldcs(reinterpret_cast<const unsigned long long*>(p + i)) : 0ull;
}

// kClear: the launch also clears words 64-bit words of clear, the state of
// the compaction that follows it, in place of a memset of its own.
template <class Op, int kIt, bool kClear = false>
__global__ void __launch_bounds__(kBlock, Op::kMinBlocks) k_lookup(const __grid_constant__ Op op, const stage_desc sd,
                                                   const uint64_t* __restrict__ probes, uint64_t m,
                                                   uint32_t* __restrict__ out, unsigned long long* clear,
                                                   uint32_t words) {
    extern __shared__ __align__(16) uint64_t cache[];
    if constexpr (Op::kStaged) stage_cache(cache, sd);
    if constexpr (kClear)
        for (uint32_t w = blockIdx.x * kBlock + threadIdx.x; w < words; w += gridDim.x * kBlock) clear[w] = 0;
    const uint64_t t0 = (uint64_t)blockIdx.x * (kBlock * kIt) + threadIdx.x;
    uint64_t next = load_probe(probes, t0, m);
#pragma unroll 1
    for (int k = 0; k < kIt; ++k) {
        const uint64_t i = t0 + (uint64_t)k * kBlock;
        if (i >= m) break;
        const uint64_t key = next;
        if (k + 1 < kIt) next = load_probe(probes, i + kBlock, m);
        __stcs(out + i, op(cache, key));
    }
}

// scattered lookup over a partitioned relation: out[rows[i]] = lookup(keys[i])
template <class Op>
constexpr int kScatterLong = std::is_same<Op, op_rs>::value ? 4 : Op::kLong;
template <class Op, int kIt>
__global__ void __launch_bounds__(kBlock, Op::kMinBlocks) k_scatter_lookup(const __grid_constant__ Op op, const stage_desc sd,
                                                           const uint64_t* __restrict__ keys,
                                                           const uint32_t* __restrict__ rows, uint64_t m,
                                                           uint32_t* __restrict__ out) {
    extern __shared__ __align__(16) uint64_t cache[];
    if constexpr (Op::kStaged) stage_cache(cache, sd);
    const uint64_t t0 = (uint64_t)blockIdx.x * (kBlock * kIt) + threadIdx.x;
    uint64_t next = load_probe(keys, t0, m);
#pragma unroll 1
    for (int k = 0; k < kIt; ++k) {
        const uint64_t i = t0 + (uint64_t)k * kBlock;
        if (i >= m) break;
        const uint64_t key = next;
        if (k + 1 < kIt) next = load_probe(keys, i + kBlock, m);
        const uint32_t r = op.template lookup<false>(cache, key);
        out[__ldcs(rows + i)] = r;
    }
}

// ---------------------------------------------------------------------------
// join pairs with decoupled look-back compaction
// ---------------------------------------------------------------------------
// Pairs are emitted in probe order.  Tiles of kBlock * items probes are
// claimed in order through an atomic counter, so every predecessor of a tile
// is already running when the tile looks back: each wait ends.  Waits are
// bounded anyway; on expiry the kernel raises the error flag (GJ_ERR_TIMEOUT
// on the host) and stops writing.
//
// From kSinglePassMin probes on, k_pairs searches and places tile by tile.
// Fewer take two passes, k_lookup with one probe a thread -- the positions go
// to the upper half of the pairs buffer (the caller provides 2m u32) -- and
// k_compact_pairs: 16,384 probes into 2^26 keys 18.7 us against 23.3 in tiles
// of four probes a thread, 2^18 probes 25 against 28, 2^20 50.1 against 49.7.
// Large calls save the positions' way through memory: 2^28 probes into a hash
// table of 2^26 keys 6631 against 6081 us, into the B+tree 6856 against 6678.
// An index in host memory keeps the two passes at every size (host_index
// below): each lookup waits on the link several times, and k_pairs' barriers
// make a whole block wait for its slowest (2^22 probes into a B+tree of 2^20
// keys 2325 us in two passes, 2692 in one).
constexpr uint64_t kSinglePassMin = 1ull << 18;
// probes a thread of k_pairs: 8 for long calls into a column that stays in L2
// (hash table of 2^20 keys 2027 against 2212 us per 2^28 probes with 4), 4
// where its sectors come from DRAM (learned index over 2^26 keys 8514 against
// 8647 with 8) and for calls too short to fill the chip with long tiles (2^18
// probes into 2^14 keys 14.8 against 18.9) or whose probes come over the host
// link (33.3 M 1697 against 1773)
constexpr int kItems = 8, kFewItems = 4;
constexpr int kCompactItems = 16;                // k_compact_pairs items per thread
static_assert(kFewItems >= 4, "the pairs scan gives each lane of a warp whole counts");
// the workspace holds one state per kStateTile probes: enough for the
// smallest tile of any pairs kernel, at the same offsets for all of them
constexpr uint32_t kStateTile = kBlock * 4;
constexpr uint32_t kCompactTile = kBlock * kCompactItems;
constexpr unsigned long long kFlagAggregate = 1ull << 62;
constexpr unsigned long long kFlagPrefix = 2ull << 62;
constexpr unsigned long long kValueMask = (1ull << 62) - 1;
constexpr uint32_t kSpinLimit = 1u << 22;

struct pairs_ws {
    unsigned long long* tile_state;  // num_tiles
    unsigned int* tile_counter;      // 1
    unsigned int* error;             // 1
    unsigned long long* totals;      // 2: pairs placed and tiles done (unordered pairs)
    uint32_t spin_limit;             // polls before a look-back gives up
};

// the workspace layout of every pairs kernel; false when it is too small
inline bool carve_pairs_ws(void* ws, size_t ws_bytes, uint64_t m, pairs_ws* pw, size_t* used) {
    const uint64_t states = (m + kStateTile - 1) / kStateTile;
    workspace_carver wc(ws, ws_bytes);
    pw->tile_state = wc.take<unsigned long long>(states ? states : 1);
    pw->tile_counter = wc.take<unsigned int>(2);
    pw->error = pw->tile_counter ? pw->tile_counter + 1 : nullptr;
    pw->totals = wc.take<unsigned long long>(2);
    pw->spin_limit = kSpinLimit;
    *used = wc.used;
    return pw->tile_state && pw->tile_counter && pw->totals;
}

// Exclusive prefix of tile `tile` (> 0) from the states of its predecessors,
// read 32 at a time by the calling warp: lane i reads tile j - i, and the
// window is summed up to its nearest published prefix.  Returns false when
// the wait ran out.
__device__ __forceinline__ bool look_back(const pairs_ws& ws, uint32_t tile, uint32_t lane,
                                          unsigned long long* prefix_out) {
    unsigned long long prefix = 0;
    int64_t j = (int64_t)tile - 1;
    uint32_t spins = 0;
    for (;;) {
        const int64_t idx = j - (int64_t)lane;
        const unsigned long long st =
            idx >= 0 ? *reinterpret_cast<volatile unsigned long long*>(&ws.tile_state[idx]) : (kFlagPrefix | 0ull);
        const unsigned long long flag = st & ~kValueMask;
        const uint32_t not_ready = __ballot_sync(0xffffffffu, flag == 0);
        const uint32_t has_prefix = __ballot_sync(0xffffffffu, flag == kFlagPrefix);
        // lanes up to (and including) the nearest prefix must all be published
        const uint32_t need = has_prefix ? (2u << (__ffs(has_prefix) - 1)) - 1u : 0xffffffffu;
        if (not_ready & need) {
            if (++spins > ws.spin_limit) return false;
            continue;
        }
        unsigned long long v = ((need >> lane) & 1u) ? (st & kValueMask) : 0ull;
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        prefix += v;
        if (has_prefix) break;
        j -= 32;
    }
    *prefix_out = prefix;
    return true;
}

// One tile of kBlock * kIt items on its way to pairs: its results (kInvalid
// for no pair; item k of thread t is probe k * kBlock + t of the tile, output
// order is probe order, i.e. (k, warp, lane) order), which lanes hold one, and
// the pairs before each (k, warp) group.
template <int kIt>
struct tile_pairs {
    static constexpr int kWarps = kBlock / 32;
    uint32_t pos[kBlock * kIt];
    uint32_t before[kIt * kWarps];
    uint32_t ballot[kIt * kWarps];
    uint32_t total;
};

// Counts the tile's pairs (each thread's own results are in t.pos) and leaves
// the exclusive scan of the groups in t.before; ends with a barrier.  publish(
// total) is called by every lane of warp 0 as soon as the total is known.
template <int kIt, class Publish>
__device__ __forceinline__ void count_tile(tile_pairs<kIt>& t, Publish&& publish) {
    constexpr int kWarps = kBlock / 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t ballot = __ballot_sync(0xffffffffu, t.pos[k * kBlock + threadIdx.x] != kInvalid);
        if (lane == 0) {
            t.before[k * kWarps + warp] = __popc(ballot);
            t.ballot[k * kWarps + warp] = ballot;
        }
    }
    __syncthreads();
    if (warp == 0) {
        constexpr int kPerLane = kIt * kWarps / 32;
        uint32_t v[kPerLane];
        uint32_t sum = 0;
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
            v[j] = t.before[lane * kPerLane + j];
            sum += v[j];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += x;
        }
        publish(__shfl_sync(0xffffffffu, incl, 31));
        uint32_t run = incl - sum;
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
            t.before[lane * kPerLane + j] = run;
            run += v[j];
        }
    }
    __syncthreads();
}

// the tile's pairs from place `first` on
template <int kIt, class RowOf>
__device__ __forceinline__ void write_tile(const tile_pairs<kIt>& t, RowOf&& row_of, uint32_t tile, uint2* pairs,
                                           uint64_t first) {
    constexpr int kWarps = kBlock / 32;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t ballot = t.ballot[k * kWarps + warp];
        if ((ballot >> lane) & 1u) {
            const uint64_t i = (uint64_t)tile * (kBlock * kIt) + (uint64_t)k * kBlock + threadIdx.x;
            const uint64_t o = first + t.before[k * kWarps + warp] + __popc(ballot & ((1u << lane) - 1u));
            const uint32_t row = row_of(k, i);
            __stcs(reinterpret_cast<unsigned long long*>(pairs + o),
                   ((unsigned long long)t.pos[k * kBlock + threadIdx.x] << 32) | row);
        }
    }
}

// ordered pairs, first half: count the tile and publish the count
template <int kIt>
__device__ __forceinline__ void publish_tile(tile_pairs<kIt>& t, uint32_t tile, const pairs_ws& ws) {
    count_tile(t, [&](unsigned long long total) {
        if ((threadIdx.x & 31) == 0) {
            t.total = (uint32_t)total;
            atomicExch(&ws.tile_state[tile], (tile == 0 ? kFlagPrefix : kFlagAggregate) | total);
        }
    });
}

// ordered pairs, second half: look back for the place of a published tile and
// write its pairs; the block's reads of t are done when it returns.  Returns
// false when the kernel must stop (look-back timed out).
template <int kIt, class RowOf>
__device__ __forceinline__ bool place_tile(const tile_pairs<kIt>& t, RowOf&& row_of, uint32_t tile, uint2* pairs,
                                           uint64_t* __restrict__ d_count, const pairs_ws& ws, uint32_t num_tiles) {
    __shared__ unsigned long long s_prefix;
    __shared__ int s_abort;
    if (threadIdx.x < 32) {
        unsigned long long prefix = 0;
        bool ok = true;
        if (tile != 0) ok = look_back(ws, tile, threadIdx.x, &prefix);
        if (threadIdx.x == 0) {
            if (!ok)
                atomicExch(ws.error, 1u);
            else if (tile != 0)
                atomicExch(&ws.tile_state[tile], kFlagPrefix | (prefix + t.total));
            s_abort = ok ? 0 : 1;
            s_prefix = prefix;
            if (ok && tile == num_tiles - 1) *d_count = prefix + t.total;
        }
    }
    __syncthreads();
    if (s_abort) return false;
    write_tile(t, row_of, tile, pairs, s_prefix);
    __syncthreads();
    return true;
}

// One tile from its results to its pairs: fill(t0, pos) writes the result of
// tile item j into pos[j]; row_of(k, i) is the probe row of item k of the
// calling thread (i = t0 + k * kBlock + thread).  Returns false when the
// kernel must stop (look-back timed out).  Unordered (kOrdered false), the
// tile's place comes from one atomicAdd instead of the look-back -- tiles
// in the order they finish, as the reference's join kernels place their
// pairs (src/tpch/tpch_14_ij.cu:371-407) -- and the last tile to finish
// writes the count.
template <int kIt, bool kOrdered = true, class Fill, class RowOf>
__device__ __forceinline__ bool pairs_tile(Fill&& fill, RowOf&& row_of, uint32_t tile, uint2* pairs,
                                           uint64_t* __restrict__ d_count, const pairs_ws& ws, uint32_t num_tiles) {
    __shared__ tile_pairs<kIt> t;
    fill((uint64_t)tile * (kBlock * kIt), t.pos);
    if constexpr (kOrdered) {
        publish_tile(t, tile, ws);
        return place_tile(t, row_of, tile, pairs, d_count, ws, num_tiles);
    } else {
        __shared__ unsigned long long s_first;
        count_tile(t, [&](unsigned long long total) {
            if (threadIdx.x == 0) {
                s_first = atomicAdd(&ws.totals[0], total);
                __threadfence();  // this tile's total is counted before it counts as done
                if (atomicAdd(&ws.totals[1], 1ull) == (unsigned long long)num_tiles - 1ull) {
                    __threadfence();
                    *d_count = atomicAdd(&ws.totals[0], 0ull);
                }
            }
        });
        write_tile(t, row_of, tile, pairs, s_first);
        __syncthreads();
        return true;
    }
}

__device__ __forceinline__ uint32_t claim_tile(const pairs_ws& ws) {
    __shared__ uint32_t s_tile;
    if (threadIdx.x == 0) s_tile = atomicAdd(ws.tile_counter, 1u);
    __syncthreads();
    return s_tile;
}

// The block that claims tile 0 writes an empty count before its own count is
// published, so that a caller's fresh counter reads 0 even where a
// look-back times out (the last tile overwrites it behind that publication).
__device__ __forceinline__ void start_count(uint32_t tile, uint64_t* d_count) {
    if (tile == 0 && threadIdx.x == 0) {
        *d_count = 0;
        __threadfence();
    }
}


// Single pass: search and place pairs tile by tile.  Unordered, a tile is
// written as soon as it is searched.  Ordered, a block publishes its tile's count, searches its next tile, and only then looks
// back for the first tile's place and writes it: the counts of the
// predecessors have arrived by then, where a block that looked back at once
// sat idle until the slowest tile before it was searched (or its probes had
// come over the host link).
// (33.3 M probes from host memory: 2109 us, 1808 with the write put off.)
// Every look-back ends: it needs the counts of earlier tiles, which their
// blocks publish before they wait for anything.
template <class Op, bool kOrdered, int kIt>
__global__ void __launch_bounds__(kBlock, Op::kMinBlocks) k_pairs(const __grid_constant__ Op op, const stage_desc sd, const uint64_t* __restrict__ probes,
                                                  uint64_t m, uint2* __restrict__ pairs,
                                                  uint64_t* __restrict__ d_count, pairs_ws ws, uint32_t num_tiles) {
    extern __shared__ __align__(16) uint64_t cache[];
    if constexpr (Op::kStaged) stage_cache(cache, sd);
    auto search = [&](uint64_t t0, uint32_t* s_pos) {
        uint64_t next = load_probe(probes, t0 + threadIdx.x, m);
#pragma unroll 1
        for (int k = 0; k < kIt; ++k) {
            const uint64_t i = t0 + (uint64_t)k * kBlock + threadIdx.x;
            const uint64_t key = next;
            if (k + 1 < kIt) next = load_probe(probes, i + kBlock, m);
            s_pos[k * kBlock + threadIdx.x] = i < m ? op(cache, key) : kInvalid;
        }
    };
    auto row_of = [&](int, uint64_t i) { return (uint32_t)i; };
    if constexpr (!kOrdered) {
        for (;;) {
            const uint32_t tile = claim_tile(ws);
            if (tile >= num_tiles) break;
            if (!pairs_tile<kIt, false>(search, row_of, tile, pairs, d_count, ws, num_tiles)) break;
        }
    } else {
        __shared__ tile_pairs<kIt> s_tile[2];
        uint32_t pending = num_tiles;  // searched tile still to be written, in the other buffer
        for (uint32_t cur = 0;; cur ^= 1) {
            const uint32_t tile = claim_tile(ws);
            if (tile < num_tiles) {
                start_count(tile, d_count);
                search((uint64_t)tile * (kBlock * kIt), s_tile[cur].pos);
                publish_tile<kIt>(s_tile[cur], tile, ws);
            }
            if (pending < num_tiles && !place_tile<kIt>(s_tile[cur ^ 1], row_of, pending, pairs, d_count, ws, num_tiles)) break;
            pending = tile;
            if (tile >= num_tiles) break;
        }
    }
}

// Second pass of the two-pass pairs: compact the positions k_lookup wrote
// to the stash into pairs at the rank of the match.  The stash is the upper
// half of the pairs buffer, so the u32 words of pair o only reach stash
// entries j <= o: a tile writes pairs only after every earlier tile
// has published its count, i.e. after every earlier tile has read its
// positions, so no position is overwritten before it is read.  (stash and
// pairs alias, so neither is __restrict__.)
__global__ void __launch_bounds__(kBlock) k_compact_pairs(const uint32_t* stash, uint64_t m, uint2* pairs,
                                                          uint64_t* __restrict__ d_count, pairs_ws ws,
                                                          uint32_t num_tiles) {
    auto load = [&](uint64_t t0, uint32_t* s_pos) {
#pragma unroll
        for (int k = 0; k < kCompactItems; ++k) {
            const uint64_t i = t0 + (uint64_t)k * kBlock + threadIdx.x;
            s_pos[k * kBlock + threadIdx.x] = i < m ? __ldcs(stash + i) : kInvalid;
        }
    };
    auto row_of = [&](int, uint64_t i) { return (uint32_t)i; };
    for (;;) {
        const uint32_t tile = claim_tile(ws);
        if (tile >= num_tiles) break;
        start_count(tile, d_count);
        if (!pairs_tile<kCompactItems>(load, row_of, tile, pairs, d_count, ws, num_tiles)) break;
    }
}

// Pairs from block-wise sorted probes.  Each tile of kSortTile probes is first
// sorted by key in shared memory -- a counting sort over kSortBuckets equal-width buckets of the
// tile's key range -- and then searched in that order: neighbouring lanes
// follow the same path through the upper index levels, and a warp-wide load
// of one sector serves all lanes that ask for it.  Pairs leave in tile order
// (sorted within a tile, in the relation's order across tiles); the order of
// equal-bucket keys inside a tile is not fixed.
constexpr int kSortItems = 4;                        // probes per thread and tile
constexpr uint32_t kSortTile = kBlock * kSortItems;  // 1024
constexpr uint32_t kSortBuckets = kSortTile;
static_assert(kStateTile <= kSortTile && kStateTile <= kBlock * kFewItems && kStateTile <= kCompactTile,
              "the workspace needs a state per tile of every pairs kernel");

__device__ __forceinline__ unsigned bit_length(uint64_t v) { return v ? 64u - (unsigned)__clzll(v) : 0u; }

// Shared memory of one sorted tile (about 21 KB with the kernels' caches).
template <class Hint>
struct sorted_tile_smem {
    static constexpr int kWarps = kBlock / 32;
    uint64_t key[kSortTile];
    uint32_t row[kSortTile];
    __align__(16) uint32_t bucket[kSortBuckets];  // read as uint4
    unsigned long long lo[kWarps], hi[kWarps];
    uint32_t wsum[kWarps];
    Hint hint;
};

// Sorts the tile keys[t0 .. t0 + tn) by key into t.key, with row_of(j) (j =
// item inside the tile) beside each in t.row, and (for an op with a tile
// hint) leaves the hint of the tile's key range in t.hint.  Ends with a
// barrier.  The caller's previous reads of t must be behind a barrier.
template <class Op, class RowOf>
__device__ __forceinline__ void sort_tile(const Op& op, const uint64_t* cache, const uint64_t* __restrict__ keys,
                                          uint64_t t0, uint32_t tn, RowOf&& row_of,
                                          sorted_tile_smem<typename tile_hint_of<Op>::type>& t) {
    constexpr int kWarps = kBlock / 32;
    constexpr bool kHinted = !std::is_same<typename tile_hint_of<Op>::type, no_tile_hint>::value;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t key[kSortItems];
    unsigned long long lo = ~0ull, hi = 0ull;
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t j = k * kBlock + threadIdx.x;
        key[k] = j < tn ? __ldcs(reinterpret_cast<const unsigned long long*>(keys) + t0 + j) : 0ull;
        if (j < tn) {
            lo = key[k] < lo ? key[k] : lo;
            hi = key[k] > hi ? key[k] : hi;
        }
    }
    // key range of the tile
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xffffffffu, lo, d);
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, hi, d);
        lo = a < lo ? a : lo;
        hi = b > hi ? b : hi;
    }
    if (lane == 0) {
        t.lo[warp] = lo;
        t.hi[warp] = hi;
    }
    for (uint32_t b = threadIdx.x; b < kSortBuckets; b += kBlock) t.bucket[b] = 0;
    __syncthreads();
    lo = t.lo[0];
    hi = t.hi[0];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) {
        lo = t.lo[w] < lo ? t.lo[w] : lo;
        hi = t.hi[w] > hi ? t.hi[w] : hi;
    }
    if constexpr (kHinted) {
        if (threadIdx.x == 0) t.hint = op.tile(cache, lo, hi);  // read after the barriers below
    }
    const unsigned used = bit_length(hi - lo);
    constexpr unsigned kBucketBits = 10;  // kSortBuckets = 2^10
    const unsigned sh = used > kBucketBits ? used - kBucketBits : 0;  // (hi - lo) >> sh < kSortBuckets
    // counting sort: ranks inside a bucket from shared-memory atomics
    uint32_t rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t j = k * kBlock + threadIdx.x;
        rank[k] = j < tn ? atomicAdd(&t.bucket[(uint32_t)((key[k] - lo) >> sh)], 1u) : 0u;
    }
    __syncthreads();
    {
        // exclusive scan of the buckets: kSortBuckets / kBlock consecutive per thread
        static_assert(kSortBuckets / kBlock == 4, "one uint4 per thread");
        uint4* sb = reinterpret_cast<uint4*>(t.bucket) + threadIdx.x;
        const uint4 c0 = sb[0];
        const uint32_t sum = c0.x + c0.y + c0.z + c0.w;
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        if (lane == 31) t.wsum[warp] = incl;
        __syncthreads();
        uint32_t run = incl - sum;
        for (int w = 0; w < (int)warp; ++w) run += t.wsum[w];
        uint4 o0;
        o0.x = run; run += c0.x;
        o0.y = run; run += c0.y;
        o0.z = run; run += c0.z;
        o0.w = run;
        sb[0] = o0;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t j = k * kBlock + threadIdx.x;
        if (j < tn) {
            const uint32_t q = t.bucket[(uint32_t)((key[k] - lo) >> sh)] + rank[k];
            t.key[q] = key[k];
            t.row[q] = row_of(j);
        }
    }
    __syncthreads();
}

// item j of a sorted tile: its search, from the tile's hint when the op has one
template <class Op>
__device__ __forceinline__ uint32_t sorted_lookup(const Op& op, const uint64_t* cache, uint64_t key,
                                                  const typename tile_hint_of<Op>::type& h) {
    if constexpr (std::is_same<typename tile_hint_of<Op>::type, no_tile_hint>::value)
        return op.template lookup<false>(cache, key);
    else
        return op.lookup_in_tile(cache, key, h);
}

// about 21 KB of shared memory per block; 6 resident blocks (40 registers),
// fewer for index kinds compiled for fewer.
template <class Op>
__global__ void __launch_bounds__(kBlock, Op::kMinBlocks < 6 ? Op::kMinBlocks : 6) k_sorted_pairs(const __grid_constant__ Op op, const stage_desc sd,
                                                         const uint64_t* __restrict__ keys, uint64_t m,
                                                         uint2* __restrict__ pairs, uint64_t* __restrict__ d_count,
                                                         pairs_ws ws, uint32_t num_tiles) {
    extern __shared__ __align__(16) uint64_t cache[];
    using hint_t = typename tile_hint_of<Op>::type;
    __shared__ sorted_tile_smem<hint_t> t;
    stage_cache(cache, sd);  // the tiles' hints read it
    auto fill = [&](uint64_t t0, uint32_t* s_pos) {
        const uint32_t tn = m - t0 < kSortTile ? (uint32_t)(m - t0) : kSortTile;
        sort_tile(op, cache, keys, t0, tn, [&](uint32_t j) { return (uint32_t)(t0 + j); }, t);
        const hint_t h = t.hint;
#pragma unroll 1
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t j = k * kBlock + threadIdx.x;
            s_pos[j] = j < tn ? sorted_lookup(op, cache, t.key[j], h) : kInvalid;
        }
    };
    auto row_of = [&](int k, uint64_t) { return t.row[k * kBlock + threadIdx.x]; };
    for (;;) {
        const uint32_t tile = claim_tile(ws);
        if (tile >= num_tiles) break;
        start_count(tile, d_count);
        if (!pairs_tile<kSortItems>(fill, row_of, tile, pairs, d_count, ws, num_tiles)) break;
    }
}

// Block-wise sorted lookup (the reference's bws_lookup,
// src/index_lookup_common.cuh:398-549): each tile of kSortTile probes is
// sorted by key, searched in that order, and the positions are put back in
// probe order through shared memory: out[i] = lookup(probes[i]).  A block
// takes kSortedLookupTiles consecutive tiles (the shared cache is staged
// once for them).
constexpr uint32_t kSortedLookupTiles = 4;
template <class Op>
__global__ void __launch_bounds__(kBlock, Op::kMinBlocks < 6 ? Op::kMinBlocks : 6) k_sorted_lookup(const __grid_constant__ Op op, const stage_desc sd,
                                                          const uint64_t* __restrict__ probes, uint64_t m,
                                                          uint32_t* __restrict__ out) {
    extern __shared__ __align__(16) uint64_t cache[];
    using hint_t = typename tile_hint_of<Op>::type;
    __shared__ sorted_tile_smem<hint_t> t;
    __shared__ uint32_t s_pos[kSortTile];
    stage_cache(cache, sd);  // the tiles' hints read it
    for (uint32_t r = 0; r < kSortedLookupTiles; ++r) {
        const uint64_t t0 = ((uint64_t)blockIdx.x * kSortedLookupTiles + r) * kSortTile;
        if (t0 >= m) break;
        const uint32_t tn = m - t0 < kSortTile ? (uint32_t)(m - t0) : kSortTile;
        sort_tile(op, cache, probes, t0, tn, [](uint32_t j) { return j; }, t);
        const hint_t h = t.hint;
#pragma unroll 1
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t j = k * kBlock + threadIdx.x;
            if (j < tn) s_pos[t.row[j]] = sorted_lookup(op, cache, t.key[j], h);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t j = k * kBlock + threadIdx.x;
            if (j < tn) __stcs(out + t0 + j, s_pos[j]);
        }
        __syncthreads();  // t and s_pos are reused by the next tile
    }
}

// ---------------------------------------------------------------------------
// dispatch helpers
// ---------------------------------------------------------------------------
stage_desc make_stage(const gj_index* idx) {
    stage_desc sd{};
    switch (idx->type) {
        case GJ_INDEX_BINARY_SEARCH:
            if (idx->bs.fence_slots) {
                sd.src0 = idx->bs.fence;
                sd.words0 = idx->bs.fence_slots;
            }
            break;
        case GJ_INDEX_BTREE:
            if (idx->bt.cached_levels) {
                sd.src0 = idx->bt.level[idx->bt.height];
                sd.words0 = idx->bt.cache_keys;
            }
            break;
        default:
            break;
    }
    return sd;
}

size_t stage_bytes(const stage_desc& sd) { return (size_t)(sd.words0 + sd.words1) * sizeof(uint64_t); }

// a kernel's staged cache (smem bytes) beside its static shared memory, which
// together may pass the 48 KB allowed without asking
template <class Kernel>
int kernel_staged(Kernel kernel, size_t smem) {
    return smem ? kernel_smem(reinterpret_cast<const void*>(kernel), smem) : GJ_OK;
}

template <class Kernel>
int grid_for(Kernel kernel, size_t smem, uint64_t work_items, int* grid) {
    device_info di;
    GJ_TRY(current_device_info(&di));
    GJ_TRY(kernel_staged(kernel, smem));
    int per_sm = 0;
    GJ_TRY(kernel_resident(reinterpret_cast<const void*>(kernel), kBlock, smem, &per_sm));
    uint64_t g = (uint64_t)di.sm_count * per_sm;
    const uint64_t need = (work_items + kBlock - 1) / kBlock;
    if (need < g) g = need ? need : 1;
    *grid = (int)g;
    return GJ_OK;
}

// What a lookup launch of items probes a thread stages, and the op that goes
// with it: a tree's levels where blocks are long, a fence always.
template <class Op>
struct staging_choice {
    Op op;
    stage_desc sd;
    size_t bytes;
};
template <class Op, class = void>
struct stages_always : std::true_type {};
template <class Op>
struct stages_always<Op, std::void_t<decltype(std::declval<Op>().unstaged())>> : std::false_type {};
// A fence is 32 KB a block, from host memory where the index lies there, so its
// blocks are long from kFenceLongProbes on (index of 2^20 keys in host memory,
// 2048- / 256-probe blocks: 2 M probes 217 / 274 us, 120,000 42 / 40).
template <class Op>
constexpr bool fence_staged = Op::kStaged && stages_always<Op>::value;
constexpr uint64_t kFenceLongProbes = 1ull << 18;
template <class Op>
staging_choice<Op> staging(const Op& op, const stage_desc& sd, int items) {
    if constexpr (!stages_always<Op>::value) {
        if (Op::kStaged && items == 1) return {op.unstaged(), stage_desc{}, 0};
    }
    return {op, sd, Op::kStaged ? stage_bytes(sd) : 0};
}

template <class Op>
int run_lookup(const Op& op, const stage_desc& sd, uint64_t n, const uint64_t* probes, uint64_t m, uint32_t* out,
               cudaStream_t s, unsigned long long* clear = nullptr, uint32_t words = 0) {
    auto launch = [&](auto kernel, int items) {
        const auto st = staging(op, sd, items);
        GJ_TRY(kernel_staged(kernel, st.bytes));
        const uint64_t tile = (uint64_t)kBlock * items;
        kernel<<<(unsigned)((m + tile - 1) / tile), kBlock, st.bytes, s>>>(st.op, st.sd, probes, m, out, clear, words);
        GJ_CUDA_TRY(cudaGetLastError());
        return (int)GJ_OK;
    };
    if constexpr (fence_staged<Op>) {
        if (m >= kFenceLongProbes)
            return clear ? launch(k_lookup<Op, Op::kLong, true>, Op::kLong) : launch(k_lookup<Op, Op::kLong>, Op::kLong);
    }
    if (clear) return launch(k_lookup<Op, 1, true>, 1);
    bool full = false;
    GJ_TRY(long_blocks(n, m, &full, kLookupLongKeys<Op>));
    full |= nodes_long<Op>(n, m);
    return full ? launch(k_lookup<Op, Op::kLong>, Op::kLong) : launch(k_lookup<Op, 1>, 1);
}

template <class Op>
int run_sorted_lookup(const Op& op, const stage_desc& sd, const uint64_t* probes, uint64_t m, uint32_t* out,
                      cudaStream_t s) {
    const size_t smem = stage_bytes(sd);
    GJ_TRY(kernel_staged(k_sorted_lookup<Op>, smem));
    const uint64_t per_block = (uint64_t)kSortTile * kSortedLookupTiles;
    const uint64_t grid = (m + per_block - 1) / per_block;
    k_sorted_lookup<Op><<<(unsigned)grid, kBlock, smem, s>>>(op, sd, probes, m, out);
    GJ_CUDA_TRY(cudaGetLastError());
    return GJ_OK;
}

template <class Op>
int run_scatter(const Op& op, const stage_desc& sd, uint64_t n, const uint64_t* keys, const uint32_t* rows,
                uint64_t m, uint32_t* out, cudaStream_t s) {
    auto launch = [&](auto kernel, int items) {
        const auto st = staging(op, sd, items);
        GJ_TRY(kernel_staged(kernel, st.bytes));
        const uint64_t tile = (uint64_t)kBlock * items;
        kernel<<<(unsigned)((m + tile - 1) / tile), kBlock, st.bytes, s>>>(st.op, st.sd, keys, rows, m, out);
        GJ_CUDA_TRY(cudaGetLastError());
        return (int)GJ_OK;
    };
    bool full = false;
    if (std::is_same<Op, op_rs>::value) full = m >= kScatterLongProbes;
    else GJ_TRY(long_blocks(n, m, &full, std::is_same<Op, op_learned>::value ? UINT64_MAX : kL2Keys));
    full |= (kNodeSearch<Op> && n <= (1ull << 25) && m >= kScatterLongProbes) ||
            (fence_staged<Op> && m >= kFenceLongProbes);
    return full ? launch(k_scatter_lookup<Op, kScatterLong<Op>>, kScatterLong<Op>) : launch(k_scatter_lookup<Op, 1>, 1);
}

template <class Op>
int run_pairs(const Op& op, const stage_desc& sd, uint64_t n, const uint64_t* probes, uint64_t m, uint32_t* pairs,
              uint64_t* d_count, void* ws, size_t ws_bytes, uint32_t* stash, cudaStream_t s, uint32_t spin_limit = 0,
              bool skip_first_tile = false, bool unordered = false, bool host_index = false) {
    pairs_ws pw;
    size_t used = 0;
    if (!carve_pairs_ws(ws, ws_bytes, m, &pw, &used)) {
        set_error("inlj pairs: workspace of %zu bytes is smaller than the %zu required", ws_bytes,
                  pairs_workspace_bytes(m));
        return GJ_ERR_WORKSPACE;
    }
    if (m == 0) {
        GJ_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
        return GJ_OK;
    }
    if (spin_limit) pw.spin_limit = spin_limit;
    device_info di;
    GJ_TRY(current_device_info(&di));
    const bool longs = nodes_two_passes<Op>(n, m, di.sm_count);
    const bool two_passes = stash && (m < kSinglePassMin || host_index || longs);
    // the state lies in whole 64-bit words at the head of the workspace
    if (two_passes && !longs) {
        GJ_TRY(run_lookup(op, sd, n, probes, m, stash, s, pw.tile_state, (uint32_t)(used / 8)));
    } else {
        GJ_CUDA_TRY(cudaMemsetAsync(ws, 0, used, s));
        if (two_passes) GJ_TRY(run_lookup(op, sd, n, probes, m, stash, s));
    }
    // test hook: the tile counter starts at 1, so tile 0 is never claimed and
    // never publishes; every later tile's look-back runs out
    if (skip_first_tile) GJ_CUDA_TRY(cudaMemsetAsync(pw.tile_counter, 1, 1, s));
    if (two_passes) {
        const uint32_t compact_tiles = (uint32_t)((m + kCompactTile - 1) / kCompactTile);
        int grid = 0;
        GJ_TRY(grid_for(k_compact_pairs, 0, (uint64_t)compact_tiles * kBlock, &grid));
        k_compact_pairs<<<grid, kBlock, 0, s>>>(stash, m, reinterpret_cast<uint2*>(pairs), d_count, pw, compact_tiles);
        GJ_CUDA_TRY(cudaGetLastError());
        return GJ_OK;
    }
    // (the tiles of ordered pairs leave no room for a tree's levels beside L1)
    const auto st = staging(op, sd, unordered ? kItems : 1);
    auto single = [&](auto kernel, uint32_t items) {
        const uint32_t num_tiles = (uint32_t)((m + kBlock * items - 1) / (kBlock * items));
        int grid = 0;
        GJ_TRY(grid_for(kernel, st.bytes, (uint64_t)num_tiles * kBlock, &grid));
        kernel<<<grid, kBlock, st.bytes, s>>>(st.op, st.sd, probes, m, reinterpret_cast<uint2*>(pairs), d_count, pw,
                                              num_tiles);
        GJ_CUDA_TRY(cudaGetLastError());
        return (int)GJ_OK;
    };
    // a short call ends with its longest chain of searches (100,000 probes into a
    // RadixSpline of 2^26 keys 52 us with 8 a thread, 30 with 4)
    if (unordered && m < (1ull << 22)) return single(k_pairs<Op, false, kFewItems>, kFewItems);
    if (unordered) return single(k_pairs<Op, false, kItems>, kItems);
    // (stash null: host buffers; a hash table's one load a search leaves less to
    // wait for: 10^8 probes into 2^26 keys with 4 / 8 a thread, uniform 2295 /
    // 2304 us, Zipf(1.25) 726 / 655)
    const bool far = n > kL2Keys && !std::is_same<Op, op_hash>::value;
    if (!stash || far || m < (1ull << 22)) return single(k_pairs<Op, true, kFewItems>, kFewItems);
    return single(k_pairs<Op, true, kItems>, kItems);
}

template <class Op>
int run_sorted_pairs(const Op& op, const stage_desc& sd, const uint64_t* probes, uint64_t m, uint32_t* pairs,
                     uint64_t* d_count, void* ws, size_t ws_bytes, cudaStream_t s) {
    const uint32_t num_tiles = (uint32_t)((m + kSortTile - 1) / kSortTile);
    pairs_ws pw;
    size_t used = 0;
    if (!carve_pairs_ws(ws, ws_bytes, m, &pw, &used)) {
        set_error("sorted pairs: workspace of %zu bytes is smaller than the %zu required", ws_bytes,
                  pairs_workspace_bytes(m));
        return GJ_ERR_WORKSPACE;
    }
    if (m == 0) {
        GJ_CUDA_TRY(cudaMemsetAsync(d_count, 0, sizeof(uint64_t), s));
        return GJ_OK;
    }
    GJ_CUDA_TRY(cudaMemsetAsync(ws, 0, used, s));
    const size_t smem = stage_bytes(sd);
    int grid = 0;
    GJ_TRY(grid_for(k_sorted_pairs<Op>, smem, (uint64_t)num_tiles * kBlock, &grid));
    k_sorted_pairs<Op><<<grid, kBlock, smem, s>>>(op, sd, probes, m, reinterpret_cast<uint2*>(pairs), d_count, pw,
                                                  num_tiles);
    GJ_CUDA_TRY(cudaGetLastError());
    return GJ_OK;
}

template <class Op>
int run_call(const Op& op, const gj_index* idx, const lookup_call& c) {
    const stage_desc sd = make_stage(idx);
    switch (c.action) {
        case lookup_action::positions: return run_lookup(op, sd, idx->n, c.keys, c.m, c.out, c.s);
        case lookup_action::scatter: return run_scatter(op, sd, idx->n, c.keys, c.rows, c.m, c.out, c.s);
        case lookup_action::pairs:
            return run_pairs(op, sd, idx->n, c.keys, c.m, c.out, c.d_count, c.ws, c.ws_bytes, c.stash, c.s, c.spin_limit,
                             c.skip_first_tile, c.unordered, idx->params.index_memory == GJ_INDEX_MEMORY_HOST);
        case lookup_action::sorted_pairs:
            return run_sorted_pairs(op, sd, c.keys, c.m, c.out, c.d_count, c.ws, c.ws_bytes, c.s);
        case lookup_action::sorted_positions: return run_sorted_lookup(op, sd, c.keys, c.m, c.out, c.s);
    }
    set_error("probe kernels: unknown action");
    return GJ_ERR_INVALID_ARGUMENT;
}

// trees of plain nodes: sorted tiles stage their levels by themselves
template <int W>
int plain_nodes_call(const gj_index* idx, const lookup_call& c) {
    const bool sorted = c.action == lookup_action::sorted_pairs || c.action == lookup_action::sorted_positions;
    if (idx->n <= kStageKeys && !sorted) return run_call(op_btree<W, true>{idx->bt}, idx, c);
    return run_call(op_btree<W>{idx->bt}, idx, c);
}

}  // namespace
}  // namespace gj
