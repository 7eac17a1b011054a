// sort.cuh - onesweep LSD radix sort and single-pass exclusive scan for sm_100a.
//
// Replaces the dynamis-sort operator (crates/dynamis-sort/src/radix.rs:321-476 with
// sort_histogram/prefix/scatter/copy.wgsl). Semantics kept: a stable LSD sort with 8-bit digits,
// the minor word's digits first and then the major word's (radix.rs:312-317), a u32 payload
// carried along. Design is new:
//   * one up-front histogram kernel counts every digit pass in a single read of the keys;
//   * each digit pass is ONE kernel: a tile of 512 or 256 threads x 8 keys ranks its keys with
//     warp __match_any_sync (stable: rounds in index order, lanes in order), publishes its digit
//     counts, and resolves its global digit prefix by decoupled look-back over earlier tiles;
//   * up to three arrays are sorted apart by the same launches (SortSource's segments);
//   * keys are staged in shared memory in digit order so the global scatter is coalesced runs.
// Tiles are claimed from an atomic counter, so a tile only waits on tiles already running.
// Every look-back wait is bounded (spin_limit polls per thread, kLookbackSpinLimit unless a caller
// lowers it); a wait that runs out sets DYN_STATUS_LOOKBACK_TIMEOUT in the status word it is given
// and the pass finishes without trapping.
#pragma once

#include <cstdint>

#include "dynamis_cuda.h"

namespace dyn {

constexpr int kSortItems = 8;
// Tiles: 512 threads (4096 keys), or 256 (2048) while every such tile has an SM of its own. A tile's
// time is its chain of eight ranking rounds, whose match instructions share the SM's four schedulers,
// so half the warps finish it sooner; past that the wide tile's fewer look-backs win. Two words with a
// payload, three digits each, us a sort, wide / narrow: 4,096 keys 80 / 56, 30,000 82 / 68, 130,000
// 97 / 76, 300,000 99 / 86, 500,000 103 / 111.
constexpr uint32_t kSortWide = 512u, kSortNarrow = 256u;
constexpr uint32_t kSortNarrowKeys = 148u * kSortNarrow * kSortItems;
__host__ __device__ __forceinline__ uint32_t sort_threads(uint32_t cap) { return cap <= kSortNarrowKeys ? kSortNarrow : kSortWide; }
__host__ __device__ __forceinline__ uint32_t sort_tiles(uint32_t keys, uint32_t threads) {
    const uint32_t tile = threads * kSortItems;
    return (keys + tile - 1u) / tile;
}
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048 values
constexpr uint32_t kLookbackSpinLimit = 1u << 22;
constexpr uint32_t kFlagAggregate = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1u;

// DYN_STATUS_* bits: dynamis_cuda.h

__device__ __forceinline__ uint32_t load_relaxed(const uint32_t* p) {
    return *reinterpret_cast<const volatile uint32_t*>(p);
}
__device__ __forceinline__ void store_relaxed(uint32_t* p, uint32_t v) {
    *reinterpret_cast<volatile uint32_t*>(p) = v;
}

// What one sort covers: one segment, or up to three that are sorted apart by the same launches (a
// segment without keys costs its launches nothing but a test). Segment s' words start at s * stride
// in the primary buffers and, packed behind those of the segments before it, in the alternate ones.
constexpr uint32_t kMaxSegments = 3;
struct SortSource {
    const uint32_t* count[kMaxSegments];  // device counts (null: n_fixed keys in the first segment)
    uint32_t segments;
    uint32_t n_fixed, cap, stride;
};
__device__ __forceinline__ uint32_t sort_count(const SortSource& s, uint32_t segment) {
    return s.count[segment] ? min(*s.count[segment], s.cap) : s.n_fixed;
}
// Tickets in flight at most (one per tile) for segments whose keys together fit `cap`.
__host__ __device__ __forceinline__ uint32_t sort_tickets(uint32_t cap, uint32_t segments, uint32_t threads) {
    return sort_tiles(cap, threads) + segments - 1u + (cap == 0u ? 1u : 0u);
}
// The tile a ticket stands for: its segment, the segment's first ticket, its keys.
struct SortTilePlace {
    uint32_t segment, first_ticket, n, packed;  // packed: the segment's first word in the alternate buffers
    bool live;
};
__device__ __forceinline__ SortTilePlace sort_place(const SortSource& s, uint32_t ticket, uint32_t threads) {
    SortTilePlace t{0u, 0u, 0u, 0u, false};
    for (uint32_t segment = 0; segment < s.segments; ++segment) {
        const uint32_t n = sort_count(s, segment), tiles = sort_tiles(n, threads);
        if (ticket < t.first_ticket + tiles) {
            t.segment = segment;
            t.n = n;
            t.live = true;
            return t;
        }
        t.first_ticket += tiles;
        t.packed += n;
    }
    return t;
}

// Counts digit occurrences for every pass of the sort in one read, and clears the look-back words of
// the tiles its passes will run. hist: segments x passes x 256 words; lookback: passes x tickets x
// 256 words; `threads`: a pass's. Digit pass p reads word (p < minor_digits ? minor : major), byte (p or p - minor_digits).
static __global__ void k_sort_histogram(const uint32_t* __restrict__ major, const uint32_t* __restrict__ minor, SortSource src,
                                        int major_digits, int minor_digits, uint32_t* __restrict__ hist,
                                        uint32_t* __restrict__ lookback, uint32_t tickets, uint32_t threads) {
    __shared__ uint32_t local[8][256];
    const int passes = major_digits + minor_digits;
    uint32_t tiles = 0u;
    for (uint32_t segment = 0; segment < src.segments; ++segment) {
        const uint32_t n = sort_count(src, segment);
        if (n == 0u) continue;
        tiles += sort_tiles(n, threads);
        if (blockIdx.x * blockDim.x >= n) continue;
        for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) (&local[0][0])[i] = 0;
        __syncthreads();
        const uint32_t* mj_in = major + (size_t)segment * src.stride;
        const uint32_t* mn_in = minor ? minor + (size_t)segment * src.stride : nullptr;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const uint32_t mj = mj_in[i], mn = mn_in ? mn_in[i] : 0u;
            for (int p = 0; p < passes; ++p) {
                uint32_t word = p < minor_digits ? mn : mj;
                int byte = p < minor_digits ? p : p - minor_digits;
                atomicAdd(&local[p][(word >> (8 * byte)) & 255u], 1u);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
            uint32_t v = (&local[0][0])[i];
            if (v) atomicAdd(&hist[(size_t)segment * passes * 256 + i], v);
        }
        __syncthreads();
    }
    const uint32_t words = tiles * 256u;
    for (int p = 0; p < passes; ++p) {
        uint32_t* lb = lookback + (size_t)p * tickets * 256u;
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) lb[i] = 0u;
    }
}

// Exclusive scans of two values a thread over the block's first 256 threads (the others hold
// zeros and get nothing they use).
__device__ __forceinline__ void scan_256(uint32_t a, uint32_t b, uint32_t* ea, uint32_t* eb, uint32_t (*sums)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t ia = a, ib = b;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t ta = __shfl_up_sync(0xFFFFFFFFu, ia, off), tb = __shfl_up_sync(0xFFFFFFFFu, ib, off);
        if (lane >= off) {
            ia += ta;
            ib += tb;
        }
    }
    if (lane == 31 && warp < 8) {
        sums[0][warp] = ia;
        sums[1][warp] = ib;
    }
    __syncthreads();
    uint32_t pa = 0u, pb = 0u;
#pragma unroll
    for (int w = 0; w < 7; ++w) {
        if (w < warp) {
            pa += sums[0][w];
            pb += sums[1][w];
        }
    }
    *ea = pa + ia - a;
    *eb = pb + ib - b;
}

// One digit pass. The sorted word is `key` (major or minor per pass); `other` rides along. Bound by
// the look-back's latency while few tiles run and by the scattered writes otherwise: a tile is 4096
// keys (half as many look-backs as 2048), the digit totals' scan happens here and not in a launch of
// its own, a thread looks back over eight tiles' words at a time, and the three arrays leave through
// one staging buffer in turn, which keeps two blocks on an SM. 1M keys of two words with a payload, six
// passes and the histogram: 116 -> 94 us.
template <bool kTwoWords, bool kPayload, uint32_t kThreads>
static __global__ void __launch_bounds__(kThreads, 1024 / kThreads)
    k_onesweep(const uint32_t* __restrict__ key_in, const uint32_t* __restrict__ other_in,
               const uint32_t* __restrict__ val_in, uint32_t* __restrict__ key_out, uint32_t* __restrict__ other_out,
               uint32_t* __restrict__ val_out, SortSource src, bool from_primary, int shift,
               const uint32_t* __restrict__ digit_totals, uint32_t passes, uint32_t* __restrict__ lookback,
               uint32_t* __restrict__ tile_counter, uint32_t* __restrict__ status, uint32_t spin_limit) {
    constexpr int kWarps = kThreads / 32;
    constexpr uint32_t kTile = kThreads * kSortItems;
    __shared__ uint32_t warp_hist[kWarps][256];
    __shared__ uint32_t tile_start[256];
    __shared__ uint32_t global_start[256];
    __shared__ uint32_t stage[kTile];
    __shared__ uint32_t sums[2][8];
    __shared__ uint32_t tile_id;

    if (threadIdx.x == 0) tile_id = atomicAdd(tile_counter, 1u);
    for (int i = threadIdx.x; i < kWarps * 256; i += kThreads) (&warp_hist[0][0])[i] = 0u;
    __syncthreads();
    const uint32_t ticket = tile_id;
    const SortTilePlace at = sort_place(src, ticket, kThreads);
    if (!at.live) return;
    const uint32_t tile_base = (ticket - at.first_ticket) * kTile;
    const uint32_t tile_n = min(kTile, at.n - tile_base);
    const size_t primary = (size_t)at.segment * src.stride;
    const size_t in = (from_primary ? primary : (size_t)at.packed) + tile_base, out = from_primary ? (size_t)at.packed : primary;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t lane_lt = (1u << lane) - 1u;

    uint32_t keys[kSortItems];
    uint32_t others[kTwoWords ? kSortItems : 1];
    uint32_t vals[kPayload ? kSortItems : 1];
    uint32_t place[kSortItems];
    // warp w owns items [w*256, (w+1)*256); round r, lane l -> item w*256 + r*32 + l
    const uint32_t first = warp * (32 * kSortItems) + lane;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) keys[r] = first + r * 32 < tile_n ? key_in[in + first + r * 32] : 0u;
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const bool valid = first + r * 32 < tile_n;
        const uint32_t digit = valid ? ((keys[r] >> shift) & 255u) : 256u;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        uint32_t before = 0;
        if (valid) before = warp_hist[warp][digit];
        __syncwarp();
        if (valid && (peers & lane_lt) == 0u) warp_hist[warp][digit] = before + __popc(peers);
        __syncwarp();
        place[r] = before + __popc(peers & lane_lt);
    }
    // the riders' loads are in flight during the look-back
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        if (kTwoWords) others[r] = first + r * 32 < tile_n ? other_in[in + first + r * 32] : 0u;
        if (kPayload) vals[r] = first + r * 32 < tile_n ? val_in[in + first + r * 32] : 0u;
    }
    __syncthreads();
    // thread d < 256 owns digit d: prefix over warps, tile count
    const uint32_t d = threadIdx.x;
    const bool owner = d < 256u;
    uint32_t count = 0u, total = 0u;
    if (owner) {
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            uint32_t c = warp_hist[w][d];
            warp_hist[w][d] = count;
            count += c;
        }
        total = digit_totals[(size_t)at.segment * passes * 256u + d];
        store_relaxed(lookback + (size_t)ticket * 256u + d, (ticket == at.first_ticket ? kFlagPrefix : kFlagAggregate) | count);
    }
    uint32_t digit_base, start;
    scan_256(total, count, &digit_base, &start, sums);
    if (owner) {
        // decoupled look-back for this digit
        uint32_t exclusive = 0;
        if (ticket != at.first_ticket) {
            constexpr int kBack = 8;
            int32_t t = (int32_t)ticket - 1;
            const int32_t last = (int32_t)at.first_ticket;
            uint32_t spins = 0;
            bool found = false;
            while (!found) {
                uint32_t words[kBack];
#pragma unroll
                for (int u = 0; u < kBack; ++u)
                    words[u] = t - u >= last ? load_relaxed(lookback + (size_t)(t - u) * 256u + d) : 0u;
                int taken = 0;
#pragma unroll
                for (int u = 0; u < kBack; ++u) {
                    if (found || taken != u) continue;
                    const uint32_t flag = words[u] & ~kValueMask;
                    if (flag == 0u) continue;
                    exclusive += words[u] & kValueMask;
                    taken = u + 1;
                    found = flag == kFlagPrefix;
                }
                t -= taken;
                if (taken == 0 && ++spins > spin_limit) {
                    atomicOr(status, DYN_STATUS_LOOKBACK_TIMEOUT);
                    break;
                }
            }
            store_relaxed(lookback + (size_t)ticket * 256u + d, kFlagPrefix | (exclusive + count));
        }
        tile_start[d] = start;
        // where digit d's keys of this tile go, less their place in the staging buffer; kept inside
        // the segment if a look-back ran out
        global_start[d] = digit_base + exclusive - start;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        if (first + r * 32 < tile_n) {
            const uint32_t digit = (keys[r] >> shift) & 255u;
            place[r] += tile_start[digit] + warp_hist[warp][digit];
            stage[place[r]] = keys[r];
        }
    }
    __syncthreads();
    uint32_t dst[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t i = threadIdx.x + r * kThreads;
        if (i < tile_n) {
            const uint32_t k = stage[i];
            dst[r] = global_start[(k >> shift) & 255u] + i;
            if (dst[r] >= at.n) dst[r] = 0xFFFFFFFFu;  // only after a look-back that ran out
            if (dst[r] < at.n) key_out[out + dst[r]] = k;
        }
    }
    auto ride = [&](const uint32_t* words, uint32_t* to) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            if (first + r * 32 < tile_n) stage[place[r]] = words[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t i = threadIdx.x + r * kThreads;
            if (i < tile_n && dst[r] < at.n) to[out + dst[r]] = stage[i];
        }
    };
    if (kTwoWords) ride(others, other_out);
    if (kPayload) ride(vals, val_out);
}

using SortPass = void (*)(const uint32_t*, const uint32_t*, const uint32_t*, uint32_t*, uint32_t*, uint32_t*, SortSource, bool, int,
                          const uint32_t*, uint32_t, uint32_t*, uint32_t*, uint32_t*, uint32_t);
template <uint32_t kThreads>
static SortPass sort_pass(bool two, bool payload) {
    return two && payload ? k_onesweep<true, true, kThreads> : two ? k_onesweep<true, false, kThreads>
           : payload ? k_onesweep<false, true, kThreads> : k_onesweep<false, false, kThreads>;
}
static inline SortPass sort_pass(bool two, bool payload, uint32_t threads) {
    return threads == kSortNarrow ? sort_pass<kSortNarrow>(two, payload) : sort_pass<kSortWide>(two, payload);
}

// Single-pass exclusive scan of u32 values (decoupled look-back over 2048-value tiles).
// Writes out[i] = sum(in[0..i)) and, from the last tile, *total = sum(in[0..n)).
static __global__ void __launch_bounds__(kScanThreads)
    k_scan_exclusive(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, const uint32_t* __restrict__ count_ptr,
                     uint32_t n_fixed, uint32_t cap, uint32_t* __restrict__ total, uint32_t* __restrict__ lookback,
                     uint32_t* __restrict__ tile_counter, uint32_t* __restrict__ status, uint32_t spin_limit) {
    __shared__ uint32_t tile_id;
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    __shared__ uint32_t tile_exclusive;
    uint32_t n = count_ptr ? min(*count_ptr, cap) : n_fixed;
    if (threadIdx.x == 0) tile_id = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint32_t tile = tile_id;
    const uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
    if (tile * kScanTile >= n) {
        if (tile == 0 && threadIdx.x == 0 && total) *total = 0u;
        return;
    }
    uint32_t v[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        uint32_t i = base + r;
        v[r] = i < n ? in[i] : 0u;
        sum += v[r];
    }
    // block scan of per-thread sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t ws = lane < kScanThreads / 32 ? warp_sums[lane] : 0u;
        uint32_t wi = ws;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wi, off);
            if (lane >= off) wi += t;
        }
        if (lane < kScanThreads / 32) warp_sums[lane] = wi - ws;
        if (lane == kScanThreads / 32 - 1) {
            uint32_t aggregate = wi;
            uint32_t exclusive = 0;
            if (tile == 0) {
                store_relaxed(&lookback[0], kFlagPrefix | aggregate);
            } else {
                store_relaxed(&lookback[tile], kFlagAggregate | aggregate);
                int32_t t = (int32_t)tile - 1;
                uint32_t spins = 0;
                while (t >= 0) {
                    uint32_t word = load_relaxed(&lookback[t]);
                    uint32_t flag = word & ~kValueMask;
                    if (flag == 0u) {
                        if (++spins > spin_limit) {
                            atomicOr(status, DYN_STATUS_LOOKBACK_TIMEOUT);
                            break;
                        }
                        continue;
                    }
                    exclusive += word & kValueMask;
                    if (flag == kFlagPrefix) break;
                    --t;
                }
                __threadfence();
                store_relaxed(&lookback[tile], kFlagPrefix | (exclusive + aggregate));
            }
            tile_exclusive = exclusive;
            if (total && (tile + 1) * kScanTile >= n) *total = exclusive + aggregate;
        }
    }
    __syncthreads();
    uint32_t run = tile_exclusive + warp_sums[warp] + (incl - sum);
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        uint32_t i = base + r;
        if (i < n) out[i] = run;
        run += v[r];
    }
}

}  // namespace dyn
