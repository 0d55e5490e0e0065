// gj_partition.cu -- range partitioning of the probe side.
//
// Replaces the fast-interconnects prefix-sum + chunked radix-partition
// kernels driven by run_on_stream (src/index_lookup_partitioning.cu:300-359).
// The reference
// partitions on key bits [max_bits - 11, max_bits) (src/index_lookup_new.cu:
// 63-67); here the partition function is a range split of the index's key
// range, partition(k) = min((k - min) >> shift, fanout - 1), so each partition
// maps onto one contiguous slice of the index and a window's lookups walk the
// index in order (the slices stay resident in the 126 MB L2).
//
// The keys are cut into tiles.  A partition pass (all on the caller's stream):
//   1. k_part_hist    per tile and partition, how many keys the tile's chunk
//                     (a run of tiles, one block's) has before the tile
//   2. k_part_base    where each chunk's keys start in each partition
//   3. k_part_scatter keys and row ids to their partition, in tile order
// and, for callers that want values back in probe order, k_part_gather.
// The windowed partitioned INLJ that drives it is in gj_partitioned.cu.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gj_lookup_kernels.cuh"  // pairs_tile and its state

namespace gj {
namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kMaxRadixBits = 12;

__device__ __forceinline__ uint32_t part_of(uint64_t key, uint64_t min_key, uint32_t shift, uint32_t fanout) {
    if (key <= min_key) return 0;
    const uint64_t p = (key - min_key) >> shift;
    return p >= fanout ? fanout - 1 : (uint32_t)p;
}

// What the passes share.  The j-th key of tile t that goes to partition p
// lands at before[t * fanout + p] + chunk_start[c * fanout + p] + part_start[p]
// + j of the relation (c: the chunk of t), all below 2^32.
struct part_tables {
    uint32_t* before;       // tiles x fanout
    uint32_t* chunk_start;  // chunks x fanout; the histogram leaves chunk counts, k_part_base their prefixes
    uint32_t* part_start;   // fanout
    uint32_t* done;         // blocks of k_part_base that are through
    const unsigned long long* stay;  // null, or a word that is not zero where the caller turned out to need no partition
    uint32_t tiles, tiles_per_chunk, chunks, fanout;
};
struct part_func {
    uint64_t min_key;
    uint32_t shift;
};

// (the word is read by every block of a pass whose keys stream through L1)
__device__ __forceinline__ bool stays(const unsigned long long* word) {
    if (!word) return false;
    unsigned long long v;
    asm("ld.global.nc.L1::evict_last.u64 %0, [%1];" : "=l"(v) : "l"(word));
    return v != 0;
}

// sub-histograms per block: warps spread their shared-memory atomics over
// several copies when the fanout is small (fewer same-address conflicts)
__host__ __device__ __forceinline__ uint32_t hist_copies(uint32_t fanout) {
    uint32_t c = 16;
    while (c > 1 && (size_t)c * fanout * sizeof(uint32_t) > 16384) c >>= 1;
    return c;
}

// One block per chunk, tile after tile; the histogram is double buffered, so
// one barrier a tile suffices.  Bound by HBM (8 bytes a key).
template <int kB, int kTile>
__global__ void __launch_bounds__(kB) k_part_hist(const uint64_t* __restrict__ keys, uint64_t m, part_func f,
                                                  part_tables t) {
    constexpr int kIt = kTile / kB;
    if (stays(t.stay)) return;
    extern __shared__ uint32_t s_hist[];  // 2 x copies x fanout, then the chunk's counts so far
    const uint32_t fanout = t.fanout, copies = hist_copies(fanout);
    uint32_t* s_run = s_hist + 2 * copies * fanout;
    for (uint32_t p = threadIdx.x; p < (2 * copies + 1) * fanout; p += kB) s_hist[p] = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) *t.done = 0;
    const uint32_t first = blockIdx.x * t.tiles_per_chunk, last = min(t.tiles, first + t.tiles_per_chunk);
    const unsigned long long* k64 = reinterpret_cast<const unsigned long long*>(keys);
    uint64_t next[kIt];
    auto load = [&](uint32_t tile) {
#pragma unroll
        for (int k = 0; k < kIt; ++k) {
            const uint64_t i = (uint64_t)tile * kTile + k * kB + threadIdx.x;
            next[k] = i < m ? __ldcs(k64 + i) : 0ull;
        }
    };
    load(first);
    __syncthreads();
    for (uint32_t tile = first; tile < last; ++tile) {
        uint32_t* buf = s_hist + (tile & 1) * copies * fanout;
        uint32_t* mine = buf + ((threadIdx.x >> 5) & (copies - 1)) * fanout;
        uint64_t key[kIt];
#pragma unroll
        for (int k = 0; k < kIt; ++k) key[k] = next[k];
        if (tile + 1 < last) load(tile + 1);
#pragma unroll
        for (int k = 0; k < kIt; ++k)
            if ((uint64_t)tile * kTile + k * kB + threadIdx.x < m)
                atomicAdd(&mine[part_of(key[k], f.min_key, f.shift, fanout)], 1u);
        __syncthreads();
        for (uint32_t p = threadIdx.x; p < fanout; p += kB) {
            uint32_t c = 0;
            for (uint32_t q = 0; q < copies; ++q) {
                c += buf[q * fanout + p];
                buf[q * fanout + p] = 0;  // for the tile after the next, behind the next barrier
            }
            const uint32_t run = s_run[p];
            __stcs(t.before + (uint64_t)tile * fanout + p, run);
            s_run[p] = run + c;
        }
    }
    __syncthreads();
    for (uint32_t p = threadIdx.x; p < fanout; p += kB) t.chunk_start[(uint64_t)blockIdx.x * fanout + p] = s_run[p];
}

// out[p] = sum of in[0..p) over count entries, by the whole block of kB threads
// (in == out is fine)
template <int kB>
__device__ __forceinline__ void block_exclusive_scan(const uint32_t* in, uint32_t* out, uint32_t count) {
    __shared__ uint32_t s_warp[kB / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t per = (count + kB - 1) / kB;
    const uint32_t begin = threadIdx.x * per;
    uint32_t sum = 0;
    for (uint32_t q = 0; q < per; ++q)
        if (begin + q < count) sum += in[begin + q];
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= (uint32_t)d) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        constexpr int kWarps = kB / 32;
        const uint32_t v = lane < kWarps ? s_warp[lane] : 0u;
        uint32_t w = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= (uint32_t)d) w += x;
        }
        if (lane < kWarps) s_warp[lane] = w - v;
    }
    __syncthreads();
    uint32_t run = s_warp[warp] + incl - sum;
    for (uint32_t q = 0; q < per; ++q)
        if (begin + q < count) {
            const uint32_t v = in[begin + q];
            out[begin + q] = run;
            run += v;
        }
}

// Chunk counts to chunk prefixes, 32 partitions a block (lane = partition, a
// warp takes a run of chunks); the last block to finish scans the partitions'
// totals into their starts.  offsets (optional): the same as 64-bit, and m.
constexpr int kBaseBlock = 1024;
__global__ void __launch_bounds__(kBaseBlock) k_part_base(part_tables t, uint64_t m, uint64_t* __restrict__ offsets) {
    constexpr uint32_t kWarps = kBaseBlock / 32;
    if (stays(t.stay)) return;
    __shared__ uint32_t s_sum[kWarps][33];
    __shared__ bool s_last;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fanout = t.fanout;
    const uint32_t p = blockIdx.x * 32 + lane;
    const uint32_t per = (t.chunks + kWarps - 1) / kWarps;
    const uint32_t c0 = min(warp * per, t.chunks), c1 = min(c0 + per, t.chunks);
    uint32_t sum = 0;
    if (p < fanout)
        for (uint32_t c = c0; c < c1; ++c) sum += t.chunk_start[(uint64_t)c * fanout + p];
    s_sum[warp][lane] = sum;
    __syncthreads();
    uint32_t run = 0;
    for (uint32_t w = 0; w < warp; ++w) run += s_sum[w][lane];
    if (p < fanout) {
        for (uint32_t c = c0; c < c1; ++c) {
            const uint32_t v = t.chunk_start[(uint64_t)c * fanout + p];
            t.chunk_start[(uint64_t)c * fanout + p] = run;
            run += v;
        }
        if (warp == kWarps - 1) t.part_start[p] = run;  // the partition's size, for the last block
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(t.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    extern __shared__ uint32_t s_part[];  // fanout
    for (uint32_t q = threadIdx.x; q < fanout; q += kBaseBlock) s_part[q] = __ldcg(t.part_start + q);
    __syncthreads();
    block_exclusive_scan<kBaseBlock>(s_part, s_part, fanout);
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < fanout; q += kBaseBlock) {
        t.part_start[q] = s_part[q];
        if (offsets) offsets[q] = s_part[q];
    }
    if (offsets && threadIdx.x == 0) offsets[fanout] = m;
}

__device__ __forceinline__ uint32_t run_start(const part_tables& t, uint32_t tile, uint32_t p) {
    return __ldcs(t.before + (uint64_t)tile * t.fanout + p) +
           __ldg(t.chunk_start + (uint64_t)(tile / t.tiles_per_chunk) * t.fanout + p) + __ldg(t.part_start + p);
}

// Scatter, one block per tile: the tile's keys are grouped by partition in
// shared memory (a counting sort whose ranks come from shared-memory
// atomics), then every partition's run is written with consecutive threads on
// consecutive addresses.  The order inside a partition follows the tiles;
// inside a tile it is not fixed.
//
// Bound by HBM (8 bytes read, 12 written a key; 10 for kInverse) where the
// runs are long, i.e. at low fanouts, and by the sectors two runs share where
// they are short.  A run ends inside a sector that the next tile's run
// completes: tiles run in order, so the two writes meet in L2 shortly after
// one another.  (With one block per chunk of consecutive tiles instead, as
// many streams were open as blocks x partitions, more lines than L2 holds at
// fanout 2^11, and each half-written sector cost a DRAM access of its own:
// 2.58 ms per 2^27 keys.)  Independent tiles also let one block's loads
// overlap another's writes on an SM without a register prefetch.
//
// kInverse: instead of row ids the relation gets each key's offset inside its
// tile (16 bits), and the tile leaves where its runs begin in its sorted
// order: what k_part_gather needs to bring results back to probe order.
template <int kB, int kIt, int kPerSM, bool kInverse>
__global__ void __launch_bounds__(kB, kPerSM) k_part_scatter(const uint64_t* __restrict__ keys, uint64_t m, part_func f,
                                                             part_tables t, uint64_t row_base,
                                                             uint64_t* __restrict__ out_keys,
                                                             uint32_t* __restrict__ out_rows, partition_inverse iv) {
    constexpr uint32_t kTile = kB * kIt;
    static_assert(kTile <= (1u << 13) && (1u << kMaxRadixBits) <= (1u << 19), "slot packing");
    if (stays(t.stay)) return;
    extern __shared__ unsigned long long s_mem[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(s_mem);            // kTile
    uint32_t* s_start = reinterpret_cast<uint32_t*>(s_mem + kTile);   // fanout: counts, then starts in the tile
    uint32_t* s_delta = s_start + t.fanout;                           // fanout: relation index less tile place
    uint16_t* s_off = reinterpret_cast<uint16_t*>(s_delta + t.fanout);  // kTile
    const uint32_t fanout = t.fanout, tile = blockIdx.x;
    const uint64_t t0 = (uint64_t)tile * kTile;
    const uint32_t tn = m - t0 < kTile ? (uint32_t)(m - t0) : kTile;
    const unsigned long long* k64 = reinterpret_cast<const unsigned long long*>(keys) + t0;
    uint64_t key[kIt];
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t j = k * kB + threadIdx.x;
        key[k] = j < tn ? __ldcs(k64 + j) : 0ull;
    }
    for (uint32_t p = threadIdx.x; p < fanout; p += kB) {
        s_start[p] = 0;
        s_delta[p] = run_start(t, tile, p);
    }
    __syncthreads();
    uint32_t slot[kIt];  // partition << 13 | rank inside the tile's partition run
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t p = part_of(key[k], f.min_key, f.shift, fanout);
        slot[k] = (uint32_t)(k * kB + threadIdx.x) < tn ? (p << 13) | atomicAdd(&s_start[p], 1u) : 0u;
    }
    __syncthreads();
    block_exclusive_scan<kB>(s_start, s_start, fanout);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t j = k * kB + threadIdx.x;
        if (j < tn) {
            const uint32_t q = s_start[slot[k] >> 13] + (slot[k] & ((1u << 13) - 1));
            s_keys[q] = key[k];
            s_off[q] = (uint16_t)j;
        }
    }
    for (uint32_t p = threadIdx.x; p < fanout; p += kB) {
        s_delta[p] -= s_start[p];
        if constexpr (kInverse) iv.start[(uint64_t)tile * fanout + p] = (uint16_t)s_start[p];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t j = k * kB + threadIdx.x;
        if (j < tn) {
            const uint64_t x = s_keys[j];
            const uint32_t d = s_delta[part_of(x, f.min_key, f.shift, fanout)] + j;
            __stcg(reinterpret_cast<unsigned long long*>(out_keys) + d, (unsigned long long)x);
            if constexpr (kInverse) __stcg(reinterpret_cast<unsigned short*>(iv.offsets) + d, s_off[j]);
            else __stcg(out_rows + d, (uint32_t)(row_base + t0 + s_off[j]));
        }
    }
}

size_t scatter_smem_bytes(uint32_t tile, uint32_t fanout) { return (size_t)tile * 10 + (size_t)fanout * 8; }

// The scatter backwards for values of the relation: out[row] = the value of
// the probe that came from row.  A tile's values are read where the scatter
// put its keys -- one run per partition, consecutive addresses -- placed in
// probe order in shared memory and written with consecutive threads on
// consecutive rows, so every sector is whole both ways.  Storing through row
// ids instead (out[rows[i]] = value) writes each output sector in as many
// pieces as it has rows, at as many different times: 2^29 positions over 2 GB
// that way took 16 of the probe pass's 23 ms.
// Bound by HBM: 2 + 4 bytes read and 4 written per probe.  One block per
// tile, not persistent: two or more blocks per SM overlap one's loads with
// the other's writes.
// values is dense per kValueTile relation entries, at a stride of twice that
// (each tile's values lie in the first half of the room its keys took).
template <int kB, int kIt, int kPerSM>
__global__ void __launch_bounds__(kB, kPerSM) k_part_gather(const uint32_t* __restrict__ values, uint64_t m,
                                                            part_tables t, partition_inverse iv,
                                                            uint32_t* __restrict__ out) {
    constexpr uint32_t kTile = kB * kIt;
    extern __shared__ unsigned long long s_mem[];
    const uint32_t fanout = t.fanout, tile = blockIdx.x;
    uint32_t* s_out = reinterpret_cast<uint32_t*>(s_mem);              // kTile
    uint32_t* s_delta = s_out + kTile;                                 // fanout
    uint16_t* s_start = reinterpret_cast<uint16_t*>(s_delta + fanout); // fanout + 2
    uint16_t* s_part = s_start + fanout + 2;                           // kTile: partition of sorted place j
    const uint64_t t0 = (uint64_t)tile * kTile;
    const uint32_t tn = m - t0 < kTile ? (uint32_t)(m - t0) : kTile;
    for (uint32_t p = threadIdx.x; p < fanout; p += kB) {
        const uint16_t at = __ldcs(iv.start + (uint64_t)tile * fanout + p);
        s_delta[p] = run_start(t, tile, p) - at;
        s_start[p] = at;
    }
    if (threadIdx.x == 0) s_start[fanout] = (uint16_t)tn;
    __syncthreads();
    for (uint32_t p = threadIdx.x >> 5; p < fanout; p += kB / 32)
        for (uint32_t j = s_start[p] + (threadIdx.x & 31); j < s_start[p + 1]; j += 32) s_part[j] = (uint16_t)p;
    __syncthreads();
    uint32_t v[kIt];
    uint16_t o[kIt];
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t j = k * kB + threadIdx.x;
        if (j < tn) {
            const uint32_t d = s_delta[s_part[j]] + j;
            v[k] = __ldcs(values + value_index(d));
            o[k] = __ldcs(iv.offsets + d);
        }
    }
#pragma unroll
    for (int k = 0; k < kIt; ++k)
        if (k * kB + threadIdx.x < tn) s_out[o[k]] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kIt; ++k) {
        const uint32_t j = k * kB + threadIdx.x;
        if (j < tn) __stcs(out + t0 + j, s_out[j]);
    }
}

// Whether a call's probes reuse the column as they come: skewed probes, whose
// keys repeat, and probes in order or nearly so, whose neighbours lie side by
// side.  Their plain search runs from L1 and L2, which is what a partition is
// for, so it would only cost (2^25 probes into 2^26 uniform keys, partitioned /
// plain: Zipf(1.25) 598 / 430 us, Zipf(1.1) 633 / 548, Zipf(1) 655 / 704,
// Zipf(0.5) 698 / 1308; sorted 724 / 427).  Taken from kReuseSample probes, in
// runs of a warp's width spread over the call: counted are the probes that fall
// on a 128-byte line of the column that another one fell on (a bitmap of hashed
// lines), and all of a run that lies within local_lines, a partition's share of
// the column.  *word: 1 where they are more than kReuseMost: 4600 of 8192 lies
// between Zipf(1.05) (3500 to 4000 on columns of 2*10^7 to 2^28 keys) and
// Zipf(1.15) (5200 to 5500); the two ways break even at 1.0 to 1.1.
// Bound by one chain of dependent loads, a search (8 us); a cluster shares the
// bitmap, a slice a block.  The launch also clears the words 64-bit words of the
// pairs' state, *word among them, in place of a memset.
constexpr int kReuseBlock = 1024, kReuseBlocks = 8;
constexpr uint32_t kReuseSample = kReuseBlocks * kReuseBlock, kReuseRuns = kReuseSample / 32;
constexpr uint32_t kReuseSliceBits = 15, kReuseMost = 4600;
__global__ void __cluster_dims__(kReuseBlocks, 1, 1) __launch_bounds__(kReuseBlock)
    k_probe_reuse(const __grid_constant__ key_start t, const uint64_t* __restrict__ col, uint32_t n,
                  const uint64_t* __restrict__ probes, uint64_t m, uint32_t local_lines, unsigned long long* state,
                  uint32_t words, unsigned long long* word) {
    __shared__ uint32_t s_seen[(1u << kReuseSliceBits) / 32];
    __shared__ uint32_t s_again;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t i = blockIdx.x * kReuseBlock + threadIdx.x;
    const uint64_t run = i >> 5;
    const uint64_t key = ld_ro(probes + run * (m - 32) / (kReuseRuns - 1) + (i & 31));
    for (uint32_t w = i; w < words; w += kReuseSample) state[w] = 0;
    for (uint32_t w = threadIdx.x; w < (1u << kReuseSliceBits) / 32; w += kReuseBlock) s_seen[w] = 0;
    if (threadIdx.x == 0) s_again = 0;
    bool eq;
    const uint32_t line = start_lower_bound<false>(t, col, n, key, &eq) >> 4;
    const uint32_t span = __reduce_max_sync(0xffffffffu, line) - __reduce_min_sync(0xffffffffu, line);
    cluster.sync();
    uint32_t again = 1;
    if (span > local_lines) {
        const uint32_t h = (line * 0x9E3779B1u) >> (32 - kReuseSliceBits - 3), bit = h & ((1u << kReuseSliceBits) - 1);
        uint32_t* seen = cluster.map_shared_rank(s_seen, h >> kReuseSliceBits);
        again = (atomicOr(seen + (bit >> 5), 1u << (bit & 31)) >> (bit & 31)) & 1u;
    }
    again = __reduce_add_sync(0xffffffffu, again);
    if ((threadIdx.x & 31) == 0) atomicAdd(cluster.map_shared_rank(&s_again, 0), again);
    cluster.sync();
    if (i == 0) *word = s_again > kReuseMost ? 1u : 0u;
}
static_assert(kReuseBlocks == 1 << 3, "a slice of the bitmap a block");

// values[i] = result of relation entry i through the index's key start table;
// neighbouring probes share its and the column's lines in L2.  Where the call
// stays with its probes as they came (stay, k_probe_reuse), of probe i.
template <bool kExact>
__global__ void __launch_bounds__(kBlock, 8) k_relation_values(const __grid_constant__ key_start t,
                                                               const uint64_t* __restrict__ col, uint32_t n,
                                                               const uint64_t* __restrict__ relation,
                                                               const uint64_t* __restrict__ probes, uint64_t m,
                                                               const unsigned long long* __restrict__ stay,
                                                               uint32_t* __restrict__ values) {
    const uint64_t i = (uint64_t)blockIdx.x * kBlock + threadIdx.x;
    if (i >= m) return;
    // the word is looked at while the relation's key is on its way: waiting for
    // it first cost 150 us of 2^28 probes' 2.5 ms
    uint64_t key = __ldcs(reinterpret_cast<const unsigned long long*>(relation) + i);
    if (stays(stay)) key = __ldcs(reinterpret_cast<const unsigned long long*>(probes) + i);
    bool eq;
    const uint32_t lb = start_lower_bound<false>(t, col, n, key, &eq);
    __stcs(values + i, (kExact ? eq : lb < n) ? lb : kInvalid);
}

// k_part_gather into ordered pairs: a block claims tiles in order, gathers a
// tile's values into probe order (they are in it where the call stayed with its
// probes) and places its pairs behind those of the tiles before it.  6 bytes
// read and up to 8 written a probe.
constexpr int kGatherItems = 16;
constexpr uint32_t kGatherTile = kBlock * kGatherItems;
__global__ void __launch_bounds__(kBlock, 6) k_gather_pairs(const uint32_t* __restrict__ values, uint64_t m,
                                                            part_tables t, partition_inverse iv,
                                                            uint2* __restrict__ pairs, uint64_t* __restrict__ d_count,
                                                            pairs_ws ws) {
    extern __shared__ unsigned long long s_mem[];
    const uint32_t fanout = t.fanout;
    uint32_t* s_delta = reinterpret_cast<uint32_t*>(s_mem);            // fanout
    uint16_t* s_start = reinterpret_cast<uint16_t*>(s_delta + fanout); // fanout + 2
    uint16_t* s_part = s_start + fanout + 2;                           // kGatherTile
    const bool stay = stays(t.stay);
    auto gather = [&](uint64_t t0, uint32_t* pos) {
        const uint32_t tile = (uint32_t)(t0 / kGatherTile);
        const uint32_t tn = m - t0 < kGatherTile ? (uint32_t)(m - t0) : kGatherTile;
        if (stay) {
#pragma unroll 8
            for (uint32_t j = threadIdx.x; j < kGatherTile; j += kBlock)
                pos[j] = j < tn ? __ldcs(values + t0 + j) : kInvalid;
            __syncthreads();
            return;
        }
        for (uint32_t p = threadIdx.x; p < fanout; p += kBlock) {
            const uint16_t at = __ldcs(iv.start + (uint64_t)tile * fanout + p);
            s_delta[p] = run_start(t, tile, p) - at;
            s_start[p] = at;
        }
        if (threadIdx.x == 0) s_start[fanout] = (uint16_t)tn;
        __syncthreads();
        for (uint32_t p = threadIdx.x >> 5; p < fanout; p += kBlock / 32)
            for (uint32_t j = s_start[p] + (threadIdx.x & 31); j < s_start[p + 1]; j += 32) s_part[j] = (uint16_t)p;
        __syncthreads();
#pragma unroll 1
        for (uint32_t j0 = threadIdx.x; j0 < kGatherTile; j0 += 8 * kBlock) {
            uint32_t v[8];
            uint16_t o[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t j = j0 + k * kBlock;
                if (j < tn) {
                    const uint32_t d = s_delta[s_part[j]] + j;
                    v[k] = __ldcs(values + d);
                    o[k] = __ldcs(iv.offsets + d);
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t j = j0 + k * kBlock;
                if (j < tn) pos[o[k]] = v[k];
                else pos[j] = kInvalid;
            }
        }
        __syncthreads();
    };
    auto row_of = [&](int, uint64_t i) { return (uint32_t)i; };
    for (;;) {
        const uint32_t tile = claim_tile(ws);
        if (tile >= t.tiles) break;
        start_count(tile, d_count);
        if (!pairs_tile<kGatherItems>(gather, row_of, tile, pairs, d_count, ws, t.tiles)) break;
    }
}

size_t gather_smem_bytes(uint32_t tile, uint32_t fanout) {
    return (size_t)tile * (4 + 2) + (size_t)fanout * 4 + ((size_t)fanout + 2) * 2;
}

// Tile geometry.  4096 keys by blocks of 512 threads, three on an SM, up to
// fanout 2^8; from 2^9 on 8192 keys (a run of the tile then still covers
// sectors), 512 threads, two on an SM, unless that leaves SMs without a tile.
// Scatter plus gather of 2^28 keys, small / large tiles: 1892 / 2013 us at
// 2^8, 2806 / 2211 at 2^9; 1024 threads on a large tile cost 2136 at 2^8 (32
// registers, spills), four small blocks an SM 1822 against 1447 at 2^5.
// All three passes of 2^28 keys at 2^5 / 2^8 / 2^11: 1543 / 1828 / 5506 us
// before, 1293 / 1475 / 2781 now.
constexpr uint32_t kWideTile = 8192, kTile = 4096;
constexpr uint32_t kWideRadixBits = 9;
constexpr int kTileBlock = 512, kHistBlock = 1024;
constexpr uint32_t kHistPerSM = 2;

struct partition_plan {
    uint32_t fanout, tile, tiles, tiles_per_chunk, chunks;
    bool wide() const { return tile == kWideTile; }
};

partition_plan plan_of(uint64_t m, uint32_t radix_bits, int sm_count, bool wide) {
    partition_plan pl;
    pl.fanout = 1u << radix_bits;
    pl.tile = wide ? kWideTile : kTile;
    pl.tiles = (uint32_t)((m + pl.tile - 1) / pl.tile);
    const uint32_t want = (uint32_t)sm_count * kHistPerSM;
    pl.tiles_per_chunk = std::max(1u, (pl.tiles + want - 1) / want);
    pl.chunks = (pl.tiles + pl.tiles_per_chunk - 1) / pl.tiles_per_chunk;
    return pl;
}

uint64_t wide_from(int sm_count) { return 2ull * sm_count * kWideTile; }

// The chunk rows of a plan's tables by the most its tiles can need: the chunk
// count itself falls where a chunk takes one more tile, the most never does.
uint32_t chunk_rows(const partition_plan& pl, int sm_count) {
    return std::min(pl.tiles, (uint32_t)sm_count * kHistPerSM);
}

partition_plan plan_partition(uint64_t m, uint32_t radix_bits, int sm_count) {
    return plan_of(m, radix_bits, sm_count, radix_bits >= kWideRadixBits && m >= wide_from(sm_count));
}

size_t plan_bytes(const partition_plan& pl, uint32_t rows) {
    return workspace_carver::need({(size_t)pl.tiles * pl.fanout * 4, (size_t)rows * pl.fanout * 4,
                                   (size_t)pl.fanout * 4, 4});
}

bool carve_tables(void* ws, size_t ws_bytes, const partition_plan& pl, part_tables* t) {
    workspace_carver wc(ws, ws_bytes);
    t->before = wc.take<uint32_t>((size_t)pl.tiles * pl.fanout);
    t->chunk_start = wc.take<uint32_t>((size_t)pl.chunks * pl.fanout);
    t->part_start = wc.take<uint32_t>(pl.fanout);
    t->done = wc.take<uint32_t>(1);
    t->tiles = pl.tiles;
    t->tiles_per_chunk = pl.tiles_per_chunk;
    t->chunks = pl.chunks;
    t->fanout = pl.fanout;
    t->stay = nullptr;
    return t->before && t->chunk_start && t->part_start && t->done;
}

template <class Kernel, class... Args>
int launch(Kernel kernel, uint32_t grid, int block, size_t smem, cudaStream_t s, Args... args) {
    if (smem > 40 * 1024)  // with the kernels' static part, near the 48 KB allowed without asking
        GJ_TRY(kernel_smem(reinterpret_cast<const void*>(kernel), smem));
    kernel<<<grid, block, smem, s>>>(args...);
    GJ_CUDA_TRY(cudaGetLastError());
    return GJ_OK;
}

}  // namespace

// The workspace of a window of m keys also serves any shorter window: tiles
// and chunk_rows only grow with m inside a tile size, and the windows of the
// other size below m need at most what wide_from keys in small tiles do.
size_t partition_ws_bytes(uint64_t m, uint32_t radix_bits, int sm_count) {
    if (m == 0) m = 1;
    const partition_plan own = plan_partition(m, radix_bits, sm_count);
    const partition_plan narrow = plan_of(std::min(m, wide_from(sm_count)), radix_bits, sm_count, false);
    return std::max(plan_bytes(own, chunk_rows(own, sm_count)), plan_bytes(narrow, chunk_rows(narrow, sm_count)));
}

int range_partition_impl(const uint64_t* d_keys, uint64_t m, uint64_t min_key, uint32_t shift, uint32_t radix_bits,
                         uint64_t row_base, uint64_t* d_out_keys, uint32_t* d_out_rows, uint64_t* d_offsets, void* ws,
                         size_t ws_bytes, cudaStream_t s, const partition_inverse* inverse,
                         const unsigned long long* stay) {
    device_info di;
    GJ_TRY(current_device_info(&di));
    const partition_plan pl = plan_partition(m ? m : 1, radix_bits, di.sm_count);
    part_tables t;
    if (!carve_tables(ws, ws_bytes, pl, &t)) {
        set_error("range partition: workspace of %zu bytes is smaller than the %zu required", ws_bytes,
                  partition_ws_bytes(m, radix_bits, di.sm_count));
        return GJ_ERR_WORKSPACE;
    }
    t.stay = stay;
    if (m == 0) {
        if (d_offsets) GJ_CUDA_TRY(cudaMemsetAsync(d_offsets, 0, ((size_t)pl.fanout + 1) * sizeof(uint64_t), s));
        return GJ_OK;
    }
    const part_func f{min_key, shift};
    const size_t hist_smem = (2 * (size_t)hist_copies(pl.fanout) + 1) * pl.fanout * sizeof(uint32_t);
    GJ_TRY(pl.wide() ? launch(k_part_hist<kHistBlock, kWideTile>, pl.chunks, kHistBlock, hist_smem, s, d_keys, m, f, t)
                     : launch(k_part_hist<kHistBlock, kTile>, pl.chunks, kHistBlock, hist_smem, s, d_keys, m, f, t));
    GJ_TRY(launch(k_part_base, (pl.fanout + 31) / 32, kBaseBlock, pl.fanout * sizeof(uint32_t), s, t, m, d_offsets));
    const size_t smem = scatter_smem_bytes(pl.tile, pl.fanout);
    const partition_inverse iv = inverse ? *inverse : partition_inverse{};
    auto scatter = [&](auto kernel, int block) {
        return launch(kernel, pl.tiles, block, smem, s, d_keys, m, f, t, row_base, d_out_keys, d_out_rows, iv);
    };
    constexpr int kWideIt = kWideTile / kTileBlock, kIt = kTile / kTileBlock;
    if (pl.wide())
        return inverse ? scatter(k_part_scatter<kTileBlock, kWideIt, 2, true>, kTileBlock)
                       : scatter(k_part_scatter<kTileBlock, kWideIt, 2, false>, kTileBlock);
    return inverse ? scatter(k_part_scatter<kTileBlock, kIt, 3, true>, kTileBlock)
                   : scatter(k_part_scatter<kTileBlock, kIt, 3, false>, kTileBlock);
}

bool carve_partition_inverse(void* ws, size_t ws_bytes, uint64_t m, uint32_t radix_bits, int sm_count,
                             partition_inverse* out) {
    const partition_plan pl = plan_partition(m ? m : 1, radix_bits, sm_count);
    workspace_carver wc(ws, ws_bytes);
    out->offsets = wc.take<uint16_t>(m);
    out->start = wc.take<uint16_t>((size_t)pl.tiles * pl.fanout);
    return out->offsets && out->start;
}

int gather_values(const uint32_t* d_values, uint64_t m, uint32_t radix_bits, void* ws, size_t ws_bytes,
                  const partition_inverse& iv, uint32_t* d_out, cudaStream_t s) {
    if (m == 0) return GJ_OK;
    device_info di;
    GJ_TRY(current_device_info(&di));
    const partition_plan pl = plan_partition(m, radix_bits, di.sm_count);
    part_tables t;
    if (!carve_tables(ws, ws_bytes, pl, &t)) {
        set_error("partition gather: workspace of %zu bytes is too small", ws_bytes);
        return GJ_ERR_WORKSPACE;
    }
    const size_t smem = gather_smem_bytes(pl.tile, pl.fanout);
    constexpr int kWideIt = kWideTile / kTileBlock, kIt = kTile / kTileBlock;
    return pl.wide() ? launch(k_part_gather<kTileBlock, kWideIt, 3>, pl.tiles, kTileBlock, smem, s, d_values, m, t, iv, d_out)
                     : launch(k_part_gather<kTileBlock, kIt, 4>, pl.tiles, kTileBlock, smem, s, d_values, m, t, iv, d_out);
}

namespace {
constexpr uint32_t kPairsRadixBits = 8;  // the most of a call's partition (small tiles)
// scratch of an ordered-pairs call by partition, behind pairs_workspace_bytes
struct pairs_scratch {
    void* tables;
    size_t table_bytes;
    uint32_t* values;
    void* inverse;
    size_t inverse_bytes;
};
// where it starts: behind the state, on the carver's boundary again (the state's
// size is not a whole number of sectors, and every store of a warp would
// straddle one more)
size_t pairs_scratch_offset(uint64_t m) { return (pairs_workspace_bytes(m) + 255) & ~size_t(255); }
size_t pairs_inverse_bytes(uint64_t m) {
    return workspace_carver::need({m * 2, (m / kTile + 1) * (2ull << kPairsRadixBits)});
}
}  // namespace

size_t pairs_partition_bytes(uint64_t m) {
    if (m < kPartitionPairsMin || m > kPartitionPairsMax) return 0;
    // no device is asked: more SMs than there are only make the tables larger
    return pairs_scratch_offset(m) - pairs_workspace_bytes(m) +
           workspace_carver::need({partition_ws_bytes(m, kPairsRadixBits, 256) + (1u << 20), m * 4,
                                   pairs_inverse_bytes(m)});
}

// Ordered pairs by way of a partition: large calls into columns far larger than
// L2, where the partition, the probes from L2 and the gather cost less than a
// random DRAM access a probe.  2^28 probes, plain / so: 2^26 uniform keys 6687 /
// 4650 us (sample 11, histogram 350, scatter 925, probes 2550, gather 840),
// lognormal 6675 / 5270; 2^24 keys 4237 / 4567.
// 2^25 probes are about where lognormal columns break even (754 / 752).  Never
// hash tables, whose plain search is one load, and no columns whose table
// windows take long searches: below 2^26 keys where those dwarf the rest (2^25
// clustered keys, 2.4 loads a search, 5505 / 5955; 2^26 8628 / 5995), and for
// the learned index, whose leaves know clustered keys.  Probes that reuse the
// column as they come take the plain search through the same table, decided on
// the device (k_probe_reuse): 2^25 probes into 2^26 keys 572 / 470 us at
// Zipf(1.25), 703 / 466 sorted, for 1.5 % of an even call of 2^25 probes and
// 0.5 % of 2^28.
//
// The relation's keys lie in the pairs buffer, which has 8 bytes a probe and is
// not written before the gather.
bool may_partition_pairs(const gj_index* idx) {
    return idx->type != GJ_INDEX_NO_OP && idx->type != GJ_INDEX_HASH && idx->in_hbm &&
           (reinterpret_cast<uintptr_t>(idx->d_col) & 31) == 0 && idx->n > partition_pairs_keys(idx->type);
}

bool partitions_pairs(const gj_index* idx) {
    const double most = idx->type == GJ_INDEX_LEARNED || idx->n < (1ull << 26) ? 2.0 : 4.0;
    return may_partition_pairs(idx) && idx->rel.pos && idx->rel_loads <= most;
}

int launch_pairs_by_partition(const gj_index* idx, const uint64_t* d_probes, uint64_t m, uint32_t* d_pairs,
                              uint64_t* d_count, void* ws, size_t ws_bytes, cudaStream_t s, bool* taken) {
    *taken = false;
    if (m < kPartitionPairsMin || m > kPartitionPairsMax || !partitions_pairs(idx)) return GJ_OK;
    const uint32_t bits = std::min(default_radix_bits(idx->n), kPairsRadixBits);
    device_info di;
    GJ_TRY(current_device_info(&di));
    const size_t head = pairs_scratch_offset(m);
    if (ws_bytes <= head) return GJ_OK;
    pairs_ws pw;
    size_t used = 0;
    if (!carve_pairs_ws(ws, head, m, &pw, &used)) return GJ_OK;
    workspace_carver wc(static_cast<char*>(ws) + head, ws_bytes - head);
    pairs_scratch sc;
    sc.table_bytes = partition_ws_bytes(m, bits, di.sm_count);
    sc.tables = wc.take<char>(sc.table_bytes);
    sc.values = wc.take<uint32_t>(m);
    sc.inverse_bytes = pairs_inverse_bytes(m);
    sc.inverse = wc.take<char>(sc.inverse_bytes);
    partition_inverse iv{};
    part_tables t;
    const partition_plan pl = plan_partition(m, bits, di.sm_count);
    if (!sc.tables || !sc.values || !sc.inverse ||
        !carve_partition_inverse(sc.inverse, sc.inverse_bytes, m, bits, di.sm_count, &iv) ||
        !carve_tables(sc.tables, sc.table_bytes, pl, &t))
        return GJ_OK;
    static_assert(kGatherTile == kTile, "the gather's tiles are the scatter's");
    *taken = true;
    uint64_t* keys = reinterpret_cast<uint64_t*>(d_pairs);
    // (the totals are the unordered pairs' words of the state, which lies in
    // whole 64-bit words at the head of the workspace)
    t.stay = pw.totals;
    GJ_TRY(launch(k_probe_reuse, kReuseBlocks, kReuseBlock, 0, s, idx->rel, idx->d_col, (uint32_t)idx->n, d_probes, m,
                  (uint32_t)(idx->n >> 4 >> bits), pw.tile_state, (uint32_t)(used / 8), pw.totals));
    GJ_TRY(range_partition_impl(d_probes, m, idx->min_key, shift_for(idx->min_key, idx->max_key, bits), bits, 0, keys,
                                nullptr, nullptr, sc.tables, sc.table_bytes, s, &iv, t.stay));
    const uint32_t blocks = (uint32_t)((m + kBlock - 1) / kBlock);
    const bool exact = idx->type == GJ_INDEX_BTREE || idx->type == GJ_INDEX_HARMONIA;
    GJ_TRY(launch(exact ? k_relation_values<true> : k_relation_values<false>, blocks, kBlock, 0, s, idx->rel, idx->d_col,
                  (uint32_t)idx->n, static_cast<const uint64_t*>(keys), d_probes, m, t.stay, sc.values));
    const size_t smem = (size_t)pl.fanout * 4 + ((size_t)pl.fanout + 2) * 2 + kGatherTile * 2;
    int grid = 0;
    GJ_TRY(grid_for(k_gather_pairs, smem, (uint64_t)pl.tiles * kBlock, &grid));
    return launch(k_gather_pairs, (uint32_t)grid, kBlock, smem, s, static_cast<const uint32_t*>(sc.values), m, t, iv,
                  reinterpret_cast<uint2*>(d_pairs), d_count, pw);
}

// key range used by the partitioned INLJ for an index (recorded at build)
void index_key_range(const gj_index* idx, uint64_t* min_key, uint64_t* max_key) {
    *min_key = idx->min_key;
    *max_key = idx->max_key;
}

uint32_t default_radix_bits(uint64_t n) {
    // about 2^21 index keys (16 MB of column, 8 MB of directory) per partition,
    // fanout within [2^5, 2^12]: a partition's slices stay in L2 while it is
    // probed, and the scatter's runs stay long.  Positions of 2^29 probes into
    // 2^28 uniform keys 9.9 / 8.8 / 9.1 / 9.8 ms at 2^5 .. 2^8, lognormal (whose
    // fullest partitions hold many times the mean) 15.5 / 12.4 / 10.5 / 10.5;
    // 2^28 into 2^26 keys 4.34 / 4.42 / 4.52 / 4.81 and 5.18 / 4.91 / 4.90 / 5.13.
    uint32_t b = 5;
    while (b < kMaxRadixBits && (n >> b) > (1ull << 21)) ++b;
    return b;
}

uint32_t shift_for(uint64_t min_key, uint64_t max_key, uint32_t radix_bits) {
    const uint64_t range = max_key - min_key;
    const unsigned used = range ? 64u - (unsigned)__builtin_clzll(range) : 0u;
    return used > radix_bits ? used - radix_bits : 0u;
}

}  // namespace gj

using namespace gj;

extern "C" {

int gj_partition_workspace_size(uint64_t m, uint32_t radix_bits, size_t* bytes) {
    GJ_CHECK_ARG(bytes, "gj_partition_workspace_size: null argument");
    GJ_CHECK_ARG(radix_bits >= 1 && radix_bits <= kMaxRadixBits, "gj_partition_workspace_size: radix_bits not in [1, 12]");
    device_info di;
    GJ_TRY(current_device_info(&di));
    *bytes = partition_ws_bytes(m, radix_bits, di.sm_count);
    return GJ_OK;
}

int gj_debug_partition_bytes(uint64_t m, uint32_t radix_bits, uint32_t sm_count, size_t* reserved, size_t* used) {
    GJ_CHECK_ARG(reserved && used, "gj_debug_partition_bytes: null argument");
    GJ_CHECK_ARG(radix_bits >= 1 && radix_bits <= kMaxRadixBits, "gj_debug_partition_bytes: radix_bits not in [1, 12]");
    GJ_CHECK_ARG(sm_count >= 1 && sm_count <= 1024, "gj_debug_partition_bytes: sm_count not in [1, 1024]");
    const partition_plan pl = plan_partition(m ? m : 1, radix_bits, (int)sm_count);
    *reserved = partition_ws_bytes(m, radix_bits, (int)sm_count);
    *used = plan_bytes(pl, pl.chunks);
    return GJ_OK;
}

int gj_range_partition(const uint64_t* d_keys, uint64_t m, uint64_t min_key, uint32_t shift, uint32_t radix_bits,
                       uint64_t* d_out_keys, uint32_t* d_out_rows, uint64_t* d_offsets, void* d_workspace,
                       size_t workspace_bytes, void* stream) {
    GJ_CHECK_ARG(radix_bits >= 1 && radix_bits <= kMaxRadixBits, "gj_range_partition: radix_bits not in [1, 12]");
    GJ_CHECK_ARG(m == 0 || (d_keys && d_out_keys && d_out_rows), "gj_range_partition: null buffer");
    GJ_CHECK_ARG(shift < 64, "gj_range_partition: shift must be < 64");
    if (m > (uint64_t)UINT32_MAX) {
        set_error("gj_range_partition: row ids must fit 32 bits");
        return GJ_ERR_TOO_LARGE;
    }
    return range_partition_impl(d_keys, m, min_key, shift, radix_bits, 0, d_out_keys, d_out_rows, d_offsets,
                                d_workspace, workspace_bytes, as_stream(stream));
}

int gj_partitioned_lookup(const gj_index* index, const uint64_t* d_part_keys, const uint32_t* d_part_rows, uint64_t m,
                          uint32_t* d_positions, void* stream) {
    GJ_CHECK_ARG(index, "gj_partitioned_lookup: null index");
    GJ_CHECK_ARG(m == 0 || (d_part_keys && d_part_rows && d_positions), "gj_partitioned_lookup: null buffer");
    return launch_scatter_lookup(index, d_part_keys, d_part_rows, m, d_positions, as_stream(stream));
}

}  // extern "C"
