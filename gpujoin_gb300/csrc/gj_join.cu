// gj_join.cu -- star-join aggregate: filter the fact table on a date window,
// look the surviving foreign keys up in the dimension index, and sum
// price * (100 - discount) overall and over flagged dimension rows.
//
// Replaces ij_plain_kernel / ij_lookup_kernel + ij_join_kernel
// (src/tpch/tpch_14_ij.cu:34-85, :371-459) with the semantics of the CPU
// query (src/tpch/cpu_only.cpp:230-275): rows pass when lo <= date < hi (the
// GPU kernels of the reference test `date >= upper`, a bug not reproduced).
//
// Each warp filters a run of fact rows and compacts the rows that pass into
// shared memory, and only then probes the index with them, so its lanes stay
// full during the lookups (the role of ij_np_lane_refill_scan_lookup,
// src/tpch/tpch_14_ij.cu:466-566).  Sums are integer, so the result does not
// depend on the order of the atomics.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "gj_internal.h"

namespace gj {
namespace {

constexpr int kJoinBlock = 256;

// the sums of the block's threads into out, one atomic each
__device__ __forceinline__ void add_sums(unsigned long long num, unsigned long long den,
                                         unsigned long long* __restrict__ out) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        num += __shfl_down_sync(0xffffffffu, num, d);
        den += __shfl_down_sync(0xffffffffu, den, d);
    }
    __shared__ unsigned long long s_num[kJoinBlock / 32], s_den[kJoinBlock / 32];
    if (lane == 0) {
        s_num[warp] = num;
        s_den[warp] = den;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0, b = 0;
        for (int w = 0; w < kJoinBlock / 32; ++w) {
            a += s_num[w];
            b += s_den[w];
        }
        if (a) atomicAdd(&out[0], a);
        if (b) atomicAdd(&out[1], b);
    }
}

// Warps work alone, each on runs of kV * 128 rows (kV 16-byte loads of dates
// a lane, all in flight).  At 6M rows and a month's window the whole call is
// a few memory latencies long: the dates, then per passing row the foreign
// key with price and discount beside it, the index, the flag.  So there are
// no block barriers on the way, one run of 1024 rows a warp covers such a
// table in one wave, and short tables take runs of 256.  (Block tiles of 4096
// rows with a block-wide scan took 15.3 us and a second, nearly empty wave.)
// kVec: the dates are 16-byte aligned.
template <class Lookup, int kV, bool kVec>
__global__ void __launch_bounds__(kJoinBlock, kV > 4 ? 5 : 6) k_star_join(
    const __grid_constant__ Lookup lookup, const uint32_t* __restrict__ fk, const uint32_t* __restrict__ date,
    const int64_t* __restrict__ price, const int64_t* __restrict__ disc, uint64_t nfact,
    const uint8_t* __restrict__ flag, uint32_t lo, uint32_t hi, unsigned long long* __restrict__ out) {
    constexpr uint32_t kRun = kV * 128;
    __shared__ uint16_t s_rows[kJoinBlock / 32][kRun];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint16_t* rows = s_rows[warp];
    unsigned long long num = 0, den = 0;
    const uint64_t step = (uint64_t)gridDim.x * (kJoinBlock / 32) * kRun;
    for (uint64_t base = ((uint64_t)blockIdx.x * (kJoinBlock / 32) + warp) * kRun; base < nfact; base += step) {
        uint32_t pass = 0;  // bit 4 k + c: row base + 128 k + 4 lane + c
        if (kVec && nfact - base >= kRun) {
            uint4 d[kV];
#pragma unroll
            for (int k = 0; k < kV; ++k)
                d[k] = __ldcs(reinterpret_cast<const uint4*>(date + base + k * 128) + lane);
#pragma unroll
            for (int k = 0; k < kV; ++k) {
                const uint32_t b = (d[k].x >= lo && d[k].x < hi ? 1u : 0u) | (d[k].y >= lo && d[k].y < hi ? 2u : 0u) |
                                   (d[k].z >= lo && d[k].z < hi ? 4u : 0u) | (d[k].w >= lo && d[k].w < hi ? 8u : 0u);
                pass |= b << (4 * k);
            }
        } else {
#pragma unroll 1
            for (int k = 0; k < 4 * kV; ++k) {
                const uint64_t i = base + (k >> 2) * 128 + 4 * lane + (k & 3);
                if (i < nfact) {
                    const uint32_t d = __ldcs(date + i);
                    pass |= (d >= lo && d < hi ? 1u : 0u) << k;
                }
            }
        }
        const uint32_t mine = __popc(pass);
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += v;
        }
        const uint32_t count = __shfl_sync(0xffffffffu, incl, 31);
        for (uint32_t o = incl - mine; pass; pass &= pass - 1, ++o) {
            const uint32_t b = __ffs(pass) - 1;
            rows[o] = (uint16_t)((b >> 2) * 128 + 4 * lane + (b & 3));
        }
        __syncwarp();
        for (uint32_t r = lane; r < count; r += 32) {
            const uint64_t i = base + rows[r];
            const uint64_t key = __ldg(fk + i);
            const int64_t p = __ldg(reinterpret_cast<const long long*>(price) + i);
            const int64_t q = __ldg(reinterpret_cast<const long long*>(disc) + i);
            const uint32_t pos = lookup(key);
            if (pos != kInvalid) {
                const int64_t summand = p * (100 - q);
                den += (unsigned long long)summand;
                if (__ldg(flag + pos)) num += (unsigned long long)summand;
            }
        }
        __syncwarp();  // the rows are overwritten by the next run
    }
    add_sums(num, den, out);
}

// The reference's pipelined order, ij_pbws (src/tpch/tpch_14_ij.cu:95-362):
// rows that pass the date filter are buffered in shared memory across the
// block's tiles until kSortBatch of them are waiting (or the rows run out);
// the batch is sorted by foreign key, probed in that order -- neighbouring
// lanes share index paths, as in the block-wise sorted probe order -- and
// aggregated.  A buffered row is (fk << 32 | row), so the sort orders by key
// (rows below 2^32).  The sums are integers and equal the unsorted kernel's.
constexpr int kSortItems = 4;
constexpr int kSortTile = kJoinBlock * kSortItems;  // rows filtered per step
constexpr int kSortBatch = 2048;                    // buffered rows that trigger a sort
constexpr int kSortCap = 4096;                      // batch + one tile, a power of two

// ascending bitonic sort of s[0, p) (p a power of two <= kSortCap) by the block
__device__ __forceinline__ void block_bitonic_sort(unsigned long long* s, uint32_t p) {
    for (uint32_t k = 2; k <= p; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t t = threadIdx.x; t < p / 2; t += kJoinBlock) {
                // the t-th pair (i, i ^ j) with bit j of i clear
                const uint32_t i = 2 * t - (t & (j - 1));
                const uint32_t l = i ^ j;
                const unsigned long long a = s[i], b = s[l];
                const bool up = (i & k) == 0;
                if ((a > b) == up) {
                    s[i] = b;
                    s[l] = a;
                }
            }
            __syncthreads();
        }
    }
}

template <class Lookup>
__global__ void __launch_bounds__(kJoinBlock) k_star_join_sorted(const __grid_constant__ Lookup lookup,
                                                                 const uint32_t* __restrict__ fk,
                                                                 const uint32_t* __restrict__ date,
                                                                 const int64_t* __restrict__ price,
                                                                 const int64_t* __restrict__ disc, uint64_t nfact,
                                                                 const uint8_t* __restrict__ flag, uint32_t lo,
                                                                 uint32_t hi, unsigned long long* __restrict__ out) {
    __shared__ unsigned long long s_buf[kSortCap];
    __shared__ uint32_t s_warp[kJoinBlock / 32];
    __shared__ uint32_t s_fill;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long num = 0, den = 0;
    const uint64_t tiles = (nfact + kSortTile - 1) / kSortTile;
    if (threadIdx.x == 0) s_fill = 0;
    __syncthreads();
    // the block's tiles: blockIdx.x, + gridDim.x, ...; one more round flushes
    for (uint64_t t = blockIdx.x;; t += gridDim.x) {
        const bool more = t < tiles;
        if (more) {
            // filter the tile and append the passing rows to the buffer
            const uint64_t base = t * kSortTile;
            uint32_t pass[kSortItems], selected = 0;
#pragma unroll
            for (int k = 0; k < kSortItems; ++k) {
                const uint64_t i = base + (uint64_t)k * kJoinBlock + threadIdx.x;
                bool ok = false;
                if (i < nfact) {
                    const uint32_t d = __ldcs(date + i);
                    ok = (d >= lo) && (d < hi);
                }
                pass[k] = ok ? 1u : 0u;
                selected += pass[k];
            }
            uint32_t incl = selected;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= (uint32_t)d) incl += v;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            if (warp == 0) {
                const uint32_t w = lane < kJoinBlock / 32 ? s_warp[lane] : 0u;
                uint32_t wi = w;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, wi, d);
                    if (lane >= (uint32_t)d) wi += v;
                }
                if (lane < kJoinBlock / 32) s_warp[lane] = wi - w;
            }
            __syncthreads();
            uint32_t o = s_fill + s_warp[warp] + incl - selected;
#pragma unroll
            for (int k = 0; k < kSortItems; ++k) {
                if (!pass[k]) continue;
                const uint64_t i = base + (uint64_t)k * kJoinBlock + threadIdx.x;
                s_buf[o++] = ((unsigned long long)__ldg(fk + i) << 32) | (uint32_t)i;
            }
            __syncthreads();
            if (threadIdx.x == kJoinBlock - 1) s_fill = o;  // the last thread's end is the new fill
            __syncthreads();
        }
        const uint32_t fill = s_fill;
        if (fill >= (uint32_t)kSortBatch || (!more && fill > 0)) {
            // sort the batch by key (padded to a power of two with the largest value)
            uint32_t p = 1;
            while (p < fill) p <<= 1;
            for (uint32_t j = fill + threadIdx.x; j < p; j += kJoinBlock) s_buf[j] = ~0ull;
            __syncthreads();
            block_bitonic_sort(s_buf, p);
            for (uint32_t j = threadIdx.x; j < fill; j += kJoinBlock) {
                const unsigned long long e = s_buf[j];
                const uint64_t key = e >> 32, i = (uint32_t)e;
                const uint32_t pos = lookup(key);
                if (pos != kInvalid) {
                    const int64_t summand = __ldg(reinterpret_cast<const long long*>(price) + i) *
                                            (100 - __ldg(reinterpret_cast<const long long*>(disc) + i));
                    den += (unsigned long long)summand;
                    if (__ldg(flag + pos)) num += (unsigned long long)summand;
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) s_fill = 0;
            __syncthreads();
        }
        if (!more) break;
    }
    add_sums(num, den, out);
}
static_assert(kSortBatch + kSortTile <= kSortCap, "a batch plus one tile fits the buffer");

// lookups of a foreign key: the position of the equal dimension key, or
// kInvalid.  Nothing is staged in shared memory: every level comes from
// global memory.
struct join_start {
    key_start t;
    const uint64_t* col;
    uint32_t n;
    __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
        bool eq;
        const uint32_t lb = start_lower_bound(t, col, n, key, &eq);
        return eq ? lb : kInvalid;
    }
};
template <int W>
struct join_btree {
    btree_view v;
    __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
        return btree_lookup<W, true, false>(v, nullptr, key);
    }
};
struct join_harmonia {
    harmonia_view v;
    __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
        return harmonia_lookup<true, false>(v, nullptr, key);
    }
};
__device__ __forceinline__ uint32_t if_equal(const uint64_t* col, uint32_t pos, uint64_t key) {
    return pos != kInvalid && ld_ro(col + pos) == key ? pos : kInvalid;
}
struct join_bs {
    bs_view v;
    __device__ __forceinline__ uint32_t operator()(uint64_t key) const {
        bs_view u = v;
        u.fence_slots = 0;  // no shared cache in this kernel
        return if_equal(v.col, bs_lookup(u, nullptr, key), key);
    }
};
struct join_rs {
    rs_view v;
    __device__ __forceinline__ uint32_t operator()(uint64_t key) const { return if_equal(v.col, rs_lookup(v, key), key); }
};

template <class Lookup>
int run_star_join_sorted(const Lookup& l, const uint32_t* fk, const uint32_t* date,
                         const int64_t* price, const int64_t* disc, uint64_t nfact, const uint8_t* flag, uint32_t lo,
                         uint32_t hi, int64_t* out, cudaStream_t s) {
    GJ_CUDA_TRY(cudaMemsetAsync(out, 0, 2 * sizeof(int64_t), s));
    if (nfact == 0) return GJ_OK;
    device_info di;
    GJ_TRY(current_device_info(&di));
    int per_sm = 0;
    GJ_TRY(kernel_resident(reinterpret_cast<const void*>(k_star_join_sorted<Lookup>), kJoinBlock, 0, &per_sm));
    uint64_t grid = (uint64_t)di.sm_count * per_sm;
    const uint64_t tiles = (nfact + kSortTile - 1) / kSortTile;
    if (grid > tiles) grid = tiles;
    k_star_join_sorted<Lookup><<<(unsigned)grid, kJoinBlock, 0, s>>>(l, fk, date, price, disc, nfact, flag, lo, hi,
                                                                     reinterpret_cast<unsigned long long*>(out));
    GJ_CUDA_TRY(cudaGetLastError());
    return GJ_OK;
}

template <class Lookup>
int run_star_join(const Lookup& l, const uint32_t* fk, const uint32_t* date, const int64_t* price,
                  const int64_t* disc, uint64_t nfact, const uint8_t* flag, uint32_t lo, uint32_t hi, int64_t* out,
                  cudaStream_t s, bool sorted = false) {
    if (sorted) return run_star_join_sorted(l, fk, date, price, disc, nfact, flag, lo, hi, out, s);
    GJ_CUDA_TRY(cudaMemsetAsync(out, 0, 2 * sizeof(int64_t), s));
    if (nfact == 0) return GJ_OK;
    device_info di;
    GJ_TRY(current_device_info(&di));
    auto launch = [&](auto kernel, uint64_t run) {
        int per_sm = 0;
        GJ_TRY(kernel_resident(reinterpret_cast<const void*>(kernel), kJoinBlock, 0, &per_sm));
        const uint64_t blocks = (nfact + run * (kJoinBlock / 32) - 1) / (run * (kJoinBlock / 32));
        const uint64_t grid = std::min<uint64_t>((uint64_t)di.sm_count * per_sm, blocks);
        kernel<<<(unsigned)grid, kJoinBlock, 0, s>>>(l, fk, date, price, disc, nfact, flag, lo, hi,
                                                     reinterpret_cast<unsigned long long*>(out));
        GJ_CUDA_TRY(cudaGetLastError());
        return (int)GJ_OK;
    };
    if ((reinterpret_cast<uintptr_t>(date) & 15) != 0)
        return launch(k_star_join<Lookup, 2, false>, 256);
    // long runs once they fill half the chip's warps
    if (nfact >= (uint64_t)di.sm_count * 24 * 1024)
        return launch(k_star_join<Lookup, 8, true>, 1024);
    return launch(k_star_join<Lookup, 2, true>, 256);
}

}  // namespace
}  // namespace gj

using namespace gj;

namespace {
int star_join(const gj_index* dim_index, const uint32_t* d_fk, const uint32_t* d_date, const int64_t* d_price,
              const int64_t* d_discount, uint64_t nfact, const uint8_t* d_dim_flag, uint32_t lo, uint32_t hi,
              int64_t* d_out, void* stream, bool sorted) {
    GJ_CHECK_ARG(dim_index && d_out, "gj_star_join_sum: null argument");
    GJ_CHECK_ARG(nfact == 0 || (d_fk && d_date && d_price && d_discount && d_dim_flag), "gj_star_join_sum: null column");
    if (sorted && nfact > (uint64_t)UINT32_MAX) {
        set_error("gj_star_join_sum_sorted: fact rows must fit 32 bits");
        return GJ_ERR_TOO_LARGE;
    }
    cudaStream_t s = as_stream(stream);
    const gj_index* idx = dim_index;
    if (idx->ks.pos)
        return run_star_join(join_start{idx->ks, idx->d_col, (uint32_t)idx->n}, d_fk, d_date, d_price, d_discount,
                             nfact, d_dim_flag, lo, hi, d_out, s, sorted);
    btree_view bt = idx->bt;
    bt.cached_levels = 0;
    harmonia_view hm = idx->hm;
    hm.cached_nodes = 0;
    hm.cached_levels = 0;
    switch (idx->type) {
        case GJ_INDEX_BTREE:
            return btree_dispatch(idx->bt.node_keys, [&](auto w) {
                return run_star_join(join_btree<decltype(w)::value>{bt}, d_fk, d_date, d_price, d_discount,
                                     nfact, d_dim_flag, lo, hi, d_out, s, sorted);
            });
        case GJ_INDEX_HARMONIA:
            return run_star_join(join_harmonia{hm}, d_fk, d_date, d_price, d_discount, nfact, d_dim_flag, lo, hi,
                                 d_out, s, sorted);
        case GJ_INDEX_BINARY_SEARCH:
            return run_star_join(join_bs{idx->bs}, d_fk, d_date, d_price, d_discount, nfact, d_dim_flag, lo, hi,
                                 d_out, s, sorted);
        case GJ_INDEX_RADIX_SPLINE:
            return run_star_join(join_rs{idx->rs}, d_fk, d_date, d_price, d_discount, nfact, d_dim_flag, lo, hi,
                                 d_out, s, sorted);
        default:
            set_error("gj_star_join_sum: the dimension index must be btree, harmonia, binary_search or radix_spline");
            return GJ_ERR_UNSUPPORTED;
    }
}
}  // namespace

extern "C" int gj_star_join_sum(const gj_index* dim_index, const uint32_t* d_fk, const uint32_t* d_date,
                                const int64_t* d_price, const int64_t* d_discount, uint64_t nfact,
                                const uint8_t* d_dim_flag, uint32_t lo, uint32_t hi, int64_t* d_out, void* stream) {
    return star_join(dim_index, d_fk, d_date, d_price, d_discount, nfact, d_dim_flag, lo, hi, d_out, stream, false);
}

extern "C" int gj_star_join_sum_sorted(const gj_index* dim_index, const uint32_t* d_fk, const uint32_t* d_date,
                                       const int64_t* d_price, const int64_t* d_discount, uint64_t nfact,
                                       const uint8_t* d_dim_flag, uint32_t lo, uint32_t hi, int64_t* d_out,
                                       void* stream) {
    return star_join(dim_index, d_fk, d_date, d_price, d_discount, nfact, d_dim_flag, lo, hi, d_out, stream, true);
}
