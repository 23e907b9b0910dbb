// sort.cu -- parallel primitives: stable LSD radix sort of (key, value) pairs, and an
// inclusive prefix sum in a single pass with decoupled look-back between tiles.
//
// Replaces algorithms::sort (source/algorithms.cpp:59-91, 4-bit digits, three
// dispatches per digit plus a recursive scan) and algorithms::prefix_sum
// (source/algorithms.cpp:93-118, recursive three-kernel block scan).
//
// Radix sort, by the list's capacity:
//  * up to 4 096 pairs: every pass in one block (k_sort_small);
//  * up to 2^18: one histogram kernel counts the digits of every pass in one read of the
//    keys; then one kernel per 8-bit digit (k_onesweep) ranks a tile of 2048 keys (8 warps x
//    8 keys per lane, warp-striped so loads coalesce), publishes the tile's digit counts,
//    looks back over earlier tiles for its global offsets and writes the tile out digit by
//    digit (6- and 7-bit digits: at every size);
//  * above: per digit a kernel that counts the tiles' digits (k_digit_count) and one that
//    ranks and writes the tiles (k_digit_scatter), without any wait on another tile.
// Stability: inside a warp the keys are ranked in index order by votes; warps are combined
// in index order; tiles in tile order.
// Every wait on another tile is bounded (kSpinLimit) and records
// APBF_FLAG_SPIN_LIMIT instead of hanging.
#include <algorithm>
#include <mutex>

#include "apbf_internal.cuh"

namespace apbf {
namespace {

constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagIncl = 2u << 30;
constexpr uint32_t kValMask = (1u << 30) - 1u;

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p) { return *(const volatile uint32_t *)p; }
__device__ __forceinline__ void st_volatile(uint32_t *p, uint32_t v) { *(volatile uint32_t *)p = v; }


// Counts the BITS-bit digits of every pass.  hist: passes x 2^BITS.
template <int BITS>
__global__ void __launch_bounds__(256) k_sort_hist(const uint32_t *__restrict__ keys, const uint32_t *d_count,
                                                   uint32_t max_count, uint32_t key_mask, int passes,
                                                   uint32_t *__restrict__ hist) {
    constexpr uint32_t NB = 1u << BITS;
    constexpr int PM = (32 + BITS - 1) / BITS;
    __shared__ uint32_t sh[PM][NB];
    for (uint32_t q = threadIdx.x; q < PM * NB; q += blockDim.x) (&sh[0][0])[q] = 0u;
    __syncthreads();
    uint32_t n = min(*d_count, max_count);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t k = keys[i] & key_mask;
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p][(k >> (BITS * p)) & (NB - 1u)], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p)
        for (uint32_t b = threadIdx.x; b < NB; b += blockDim.x)
            if (sh[p][b]) atomicAdd(&hist[p * NB + b], sh[p][b]);
}

// Exclusive scan over the first NB threads of a block (NB a multiple of 32, at most 256);
// every thread calls it.
template <uint32_t NB>
__device__ __forceinline__ uint32_t scan_digits(uint32_t v, uint32_t *s_part) {
    const uint32_t t = threadIdx.x, l = t & 31u, w = t >> 5;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if ((int)l >= off) x += y;
    }
    if (t < NB && l == 31u) s_part[w] = x;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (uint32_t k = 0; k < NB / 32u; ++k)
        if (k < w) before += s_part[k];
    __syncthreads();  // s_part may be used again
    return before + x - v;
}

// Ranks one warp-striped chunk of keys (ITEMS per lane, in index order) by their digits:
// rank[k] = keys of the same digit before it in the warp's chunk; cnt[digit] ends as the
// chunk's digit counts.  Items past the end carry a digit of NB or more, counted nowhere.
// The lanes of equal digit are found by a vote per digit bit: __match_any_sync takes 66
// cycles of its unit for 32 different digits and kept that busy for half of a pass.
template <uint32_t NB, int ITEMS, typename C>
__device__ __forceinline__ void rank_digits(const uint32_t (&digit)[ITEMS], uint32_t (&rank)[ITEMS], C *cnt) {
    const uint32_t l = threadIdx.x & 31u, lt = (1u << l) - 1u;
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const bool valid = digit[k] < NB;
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (uint32_t bit = 1u; bit < NB; bit <<= 1) {
            const bool set = (digit[k] & bit) != 0u;
            const uint32_t with = __ballot_sync(0xffffffffu, set);
            peers &= set ? with : ~with;
        }
        const uint32_t before = valid ? (uint32_t)cnt[digit[k]] : 0u;
        rank[k] = before + __popc(peers & lt);
        __syncwarp();
        if (valid && (uint32_t)(__ffs(peers) - 1) == l) cnt[digit[k]] = (C)(before + __popc(peers));
        __syncwarp();
    }
}

// Writes a ranked tile out digit by digit: through shared memory, so that a digit's run
// leaves as whole lines.  off: where a digit's keys start in the sorted tile, base: and in
// the output, less that; warp_off: the warp's first of each digit.
template <uint32_t NB>
__device__ __forceinline__ void write_tile(const uint32_t (&keys)[kSortItems], const uint32_t (&vals)[kSortItems],
                                           const uint32_t (&digit)[kSortItems], const uint32_t (&rank)[kSortItems],
                                           const uint32_t *warp_off, const uint32_t *off, const uint32_t *base,
                                           uint32_t *s_keys, uint32_t *s_vals, uint32_t here, uint32_t key_mask,
                                           int shift, uint32_t *__restrict__ kout, uint32_t *__restrict__ vout) {
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        if (digit[k] >= NB) continue;
        const uint32_t pos = off[digit[k]] + warp_off[digit[k]] + rank[k];
        s_keys[pos] = keys[k];
        s_vals[pos] = vals[k];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = (uint32_t)k * kSortThreads + threadIdx.x;
        if (idx >= here) break;
        const uint32_t key = s_keys[idx];
        const uint32_t pos = base[((key & key_mask) >> shift) & (NB - 1u)] + idx;
        kout[pos] = key;
        vout[pos] = s_vals[idx];
    }
}

// One BITS-bit digit pass.  tile_status: tiles x 2^BITS words (flag << 30 | count).
// Thread t < 2^BITS owns digit t.
//
// Bound by latency: a tile's chain is its ticket, its keys, the ranking, the look-back and
// the scatter, so the tiles are small (2 048 keys), the look-back reads eight earlier tiles
// at a time (4 096 keys or 16 and 32 tiles at a time were slower), and the keys go through
// shared memory so that a digit's run leaves as whole lines.  Nine to seven microseconds a
// pass from 30 000 to 260 000 pairs.  A digit that all keys share (the histogram has them in
// one bin) moves none: the tile is copied, without ranks and look-back.
// (kin and vin are not __restrict__: their loads must stay behind the wait.)
constexpr int kLookBack = 8;
template <int BITS>
__global__ void __launch_bounds__(kSortThreads) k_onesweep(const uint32_t *kin, const uint32_t *vin,
                                                  uint32_t *__restrict__ kout, uint32_t *__restrict__ vout,
                                                  const uint32_t *d_count, uint32_t max_count, uint32_t key_mask,
                                                  int shift, const uint32_t *__restrict__ hist,
                                                  uint32_t *tile_counter, uint32_t *tile_status, Status *st) {
    constexpr uint32_t NB = 1u << BITS;
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_cnt[kSortWarps][NB];
    __shared__ uint32_t s_off[NB];   // where a digit's keys start in the sorted tile
    __shared__ uint32_t s_base[NB];  // and in the output, less that
    __shared__ uint32_t s_part[8];
    __shared__ uint32_t s_keys[kSortTile], s_vals[kSortTile];

    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    const bool owner = (uint32_t)t < NB;
    if (t == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (uint32_t k = t; k < kSortWarps * NB; k += kSortThreads) (&s_cnt[0][0])[k] = 0u;
    const uint32_t hist_t = owner ? __ldcg(hist + t) : 0u;
    const uint32_t n = min(*d_count, max_count);
    const uint32_t ntiles = (n + kSortTile - 1) / kSortTile;
    const bool shared_digit = __syncthreads_or(owner && hist_t == n);
    // up to here nothing that the pass before writes: its blocks end as these start
    grid_dependency_wait();
    grid_dependency_trigger();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) return;
    const uint32_t first = tile * kSortTile, here = min(n - first, (uint32_t)kSortTile);

    uint32_t keys[kSortItems], vals[kSortItems], digit[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = (uint32_t)w * (32 * kSortItems) + k * 32 + l;
        const bool valid = idx < here;
        keys[k] = valid ? kin[first + idx] : 0u;
        vals[k] = valid ? vin[first + idx] : 0u;
        digit[k] = valid ? ((keys[k] & key_mask) >> shift) & (NB - 1u) : NB + (uint32_t)l;
    }
    if (shared_digit) {
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) {
            const uint32_t idx = (uint32_t)w * (32 * kSortItems) + k * 32 + l;
            if (idx >= here) break;
            kout[first + idx] = keys[k];
            vout[first + idx] = vals[k];
        }
        return;
    }
    rank_digits<NB>(digit, rank, s_cnt[w]);
    __syncthreads();
    // thread t owns digit t: warp exclusive offsets and the tile total, published at once
    uint32_t run = 0;
    if (owner) {
#pragma unroll
        for (int k = 0; k < kSortWarps; ++k) {
            const uint32_t c = s_cnt[k][t];
            s_cnt[k][t] = run;
            run += c;
        }
        st_volatile(tile_status + (size_t)tile * NB + t, (tile == 0 ? kFlagIncl : kFlagAgg) | run);
    }
    const uint32_t off = scan_digits<NB>(run, s_part);
    const uint32_t digit_excl = scan_digits<NB>(hist_t, s_part);  // same in every tile
    if (owner) {
        s_off[t] = off;
        uint32_t excl = 0;
        int j = (int)tile - 1;
        uint32_t spins = 0;
        bool inject;
        const uint32_t limit = wait_limit(st, kSpinLimit, inject);
        while (j >= 0) {
            uint32_t v[kLookBack];
#pragma unroll
            for (int u = 0; u < kLookBack; ++u)
                v[u] = j - u >= 0 ? ld_volatile(tile_status + (size_t)(j - u) * NB + t) : kFlagIncl;
            bool open = false;  // reached a tile that has not published yet
            int passed = 0;
#pragma unroll
            for (int u = 0; u < kLookBack; ++u) {
                if (open || j < 0) continue;
                const uint32_t f = inject ? 0u : (v[u] & ~kValMask);
                if (f == 0u) {
                    open = true;
                    continue;
                }
                excl += v[u] & kValMask;
                if (f == kFlagIncl) j = -1;
                else ++passed;
            }
            if (j >= 0) j -= passed;
            if (open) {
                if (++spins > limit) {
                    set_flag(st, APBF_FLAG_SPIN_LIMIT);
                    st->spin_where = 1u;
                    break;
                }
                __nanosleep(32);
            }
        }
        if (tile != 0) st_volatile(tile_status + (size_t)tile * NB + t, kFlagIncl | ((excl + run) & kValMask));
        s_base[t] = digit_excl + excl - off;
    }
    __syncthreads();
    write_tile<NB>(keys, vals, digit, rank, s_cnt[w], s_off, s_base, s_keys, s_vals, here, key_mask, shift, kout, vout);
}

// The same digit pass without any wait, for lists above kWaitFree keys (a million pairs of
// 30 bits: 58 us, with the look-back 105, 122 before either): k_digit_count
// leaves the digit counts of every tile and, added up, of every group of kSortGroup tiles;
// k_digit_scatter's tile reads the groups and the tiles of its own group in one round of
// loads while its keys arrive.  The look-back's chain grows with the number of tiles (they
// all run at once and read back eight at a time); this does not.  The keys that the scatter
// ranks are older than the counts, so it loads and ranks them while the counts are taken and
// waits for these only then (74 us without).
template <int BITS>
__global__ void __launch_bounds__(kSortThreads) k_digit_count(const uint32_t *kin, const uint32_t *d_count,
                                                              uint32_t max_count, uint32_t key_mask, int shift,
                                                              uint32_t *__restrict__ tile_counts,
                                                              uint32_t *__restrict__ group_counts) {
    constexpr uint32_t NB = 1u << BITS;
    __shared__ uint32_t s_cnt[NB];
    const uint32_t n = min(*d_count, max_count), t = threadIdx.x, tile = blockIdx.x;
    if (t < NB) s_cnt[t] = 0u;
    grid_dependency_wait();  // (every block, so that this kernel ends behind the one before it)
    grid_dependency_trigger();
    if (tile * (uint32_t)kSortTile >= n) return;
    __syncthreads();
    const uint32_t first = tile * kSortTile, here = min(n - first, (uint32_t)kSortTile);
    uint32_t key[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = (uint32_t)k * kSortThreads + t;
        key[k] = idx < here ? kin[first + idx] : 0u;
    }
#pragma unroll
    for (int k = 0; k < kSortItems; ++k)
        if ((uint32_t)k * kSortThreads + t < here) atomicAdd(&s_cnt[((key[k] & key_mask) >> shift) & (NB - 1u)], 1u);
    __syncthreads();
    if (t < NB) {
        const uint32_t c = s_cnt[t];
        tile_counts[(size_t)tile * NB + t] = c;
        if (c) atomicAdd(&group_counts[(size_t)(tile / kSortGroup) * NB + t], c);
    }
}

template <int BITS>
__global__ void __launch_bounds__(kSortThreads) k_digit_scatter(const uint32_t *__restrict__ kin,
                                                                const uint32_t *__restrict__ vin,
                                                                uint32_t *__restrict__ kout, uint32_t *__restrict__ vout,
                                                                const uint32_t *d_count, uint32_t max_count,
                                                                uint32_t key_mask, int shift,
                                                                const uint32_t *tile_counts,
                                                                const uint32_t *group_counts) {
    constexpr uint32_t NB = 1u << BITS;
    __shared__ uint32_t s_cnt[kSortWarps][NB];
    __shared__ uint32_t s_off[NB], s_base[NB], s_part[8];
    __shared__ uint32_t s_keys[kSortTile], s_vals[kSortTile];
    const uint32_t n = min(*d_count, max_count), t = threadIdx.x, w = t >> 5, l = t & 31u, tile = blockIdx.x;
    const uint32_t first = tile * kSortTile;
    const uint32_t here = first < n ? min(n - first, (uint32_t)kSortTile) : 0u;
    uint32_t keys[kSortItems], vals[kSortItems], digit[kSortItems], rank[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = w * (32 * kSortItems) + k * 32 + l;
        keys[k] = idx < here ? __ldcg(kin + first + idx) : 0u;
        vals[k] = idx < here ? __ldcg(vin + first + idx) : 0u;
    }
    for (uint32_t k = t; k < kSortWarps * NB; k += kSortThreads) (&s_cnt[0][0])[k] = 0u;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; ++k) {
        const uint32_t idx = w * (32 * kSortItems) + k * 32 + l;
        digit[k] = idx < here ? ((keys[k] & key_mask) >> shift) & (NB - 1u) : NB + l;
    }
    rank_digits<NB>(digit, rank, s_cnt[w]);
    grid_dependency_wait();  // the counts, and every block that read where this one writes
    grid_dependency_trigger();
    if (here == 0u) return;
    // the digit's keys in all tiles, and in the tiles before this one
    uint32_t all = 0, before = 0;
    if (t < NB) {
        const uint32_t groups = (n + kSortTile * kSortGroup - 1) / (kSortTile * kSortGroup), own = tile / kSortGroup;
#pragma unroll 8
        for (uint32_t g = 0; g < groups; ++g) {
            const uint32_t c = group_counts[(size_t)g * NB + t];
            all += c;
            before += g < own ? c : 0u;
        }
#pragma unroll 8
        for (uint32_t k = own * kSortGroup; k < tile; ++k) before += tile_counts[(size_t)k * NB + t];
    }
    __syncthreads();
    uint32_t run = 0;
    if (t < NB) {
#pragma unroll
        for (int k = 0; k < kSortWarps; ++k) {
            const uint32_t c = s_cnt[k][t];
            s_cnt[k][t] = run;
            run += c;
        }
    }
    const uint32_t off = scan_digits<NB>(run, s_part);
    const uint32_t digit_excl = scan_digits<NB>(all, s_part);
    if (t < NB) {
        s_off[t] = off;
        s_base[t] = digit_excl + before - off;
    }
    __syncthreads();
    write_tile<NB>(keys, vals, digit, rank, s_cnt[w], s_off, s_base, s_keys, s_vals, here, key_mask, shift, kout, vout);
}
constexpr uint32_t kWaitFree = 1u << 18;

// Every 8-bit pass of a short list in one block: the pairs stay in registers and shared
// memory between the passes.  One launch (14 us at 4 096 pairs of 21 bits, 44 us before)
// instead of a histogram, a clear and a launch per digit, whose latencies are all that a
// short sort costs.  With four times the threads and pairs it took 41 us at 5 000 pairs and 49
// at 16 384, the overlapped tiles 23 and 25.
constexpr int kSmallThreads = 256, kSmallItems = 16;
constexpr uint32_t kSmallKeys = kSmallThreads * kSmallItems;
struct SmallSort {
    uint32_t keys[kSmallKeys], vals[kSmallKeys];
    uint16_t cnt[kSmallThreads / 32][256];
    uint32_t off[256], part[8];
};
__global__ void __launch_bounds__(kSmallThreads) k_sort_small(const uint32_t *kin, const uint32_t *vin, uint32_t *kout,
                                                        uint32_t *vout, const uint32_t *d_count, uint32_t max_count,
                                                        uint32_t key_mask, int passes) {
    extern __shared__ unsigned char s_raw[];
    SmallSort &s = *reinterpret_cast<SmallSort *>(s_raw);
    grid_dependency_wait();
    grid_dependency_trigger();
    const uint32_t t = threadIdx.x, w = t >> 5, l = t & 31u;
    const uint32_t n = min(*d_count, max_count);
    uint32_t keys[kSmallItems], vals[kSmallItems], digit[kSmallItems], rank[kSmallItems];
#pragma unroll
    for (int k = 0; k < kSmallItems; ++k) {
        const uint32_t idx = w * (32 * kSmallItems) + k * 32 + l;
        keys[k] = idx < n ? kin[idx] : 0u;
        vals[k] = idx < n ? vin[idx] : 0u;
    }
    for (int p = 0; p < passes; ++p) {
        for (uint32_t k = t; k < kSmallThreads / 32 * 128; k += kSmallThreads) reinterpret_cast<uint32_t *>(&s.cnt[0][0])[k] = 0u;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSmallItems; ++k) {
            const uint32_t idx = w * (32 * kSmallItems) + k * 32 + l;
            digit[k] = idx < n ? ((keys[k] & key_mask) >> (8 * p)) & 255u : 256u + l;
        }
        rank_digits<256u>(digit, rank, s.cnt[w]);
        __syncthreads();
        uint32_t run = 0;
        if (t < 256u)
            for (int k = 0; k < kSmallThreads / 32; ++k) {
                const uint32_t c = s.cnt[k][t];
                s.cnt[k][t] = (uint16_t)run;
                run += c;
            }
        const uint32_t off = scan_digits<256u>(run, s.part);
        if (t < 256u) s.off[t] = off;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSmallItems; ++k) {
            if (digit[k] >= 256u) continue;
            const uint32_t pos = s.off[digit[k]] + s.cnt[w][digit[k]] + rank[k];
            s.keys[pos] = keys[k];
            s.vals[pos] = vals[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kSmallItems; ++k) {
            const uint32_t idx = w * (32 * kSmallItems) + k * 32 + l;
            if (idx >= n) continue;
            keys[k] = s.keys[idx];
            vals[k] = s.vals[idx];
            if (p == passes - 1) {
                kout[idx] = keys[k];
                vout[idx] = vals[k];
            }
        }
    }
}

// Single-pass inclusive scan with decoupled look-back; tile = 256 threads x 16.
constexpr int kScanItems = 16;
constexpr int kScanTile = 256 * kScanItems;

__global__ void __launch_bounds__(256) k_scan(uint32_t *data, const uint32_t *d_count, uint32_t max_count,
                                              uint32_t *tile_counter, uint32_t *tile_status, Status *st) {
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_excl;
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    if (t == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const uint32_t n = min(*d_count, max_count);
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    const uint32_t tile = s_tile;
    if (tile >= ntiles) return;
    // blocked arrangement: thread t owns items [t*16, t*16+16) of the tile
    const uint32_t base = tile * kScanTile + (uint32_t)t * kScanItems;
    uint32_t v[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        uint32_t idx = base + k;
        v[k] = idx < n ? data[idx] : 0u;
        sum += v[k];
        v[k] = sum;  // thread-local inclusive
    }
    // block exclusive scan of thread sums
    uint32_t x = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (l >= off) x += y;
    }
    if (l == 31) s_warp[w] = x;
    __syncthreads();
    if (t < 32) {
        uint32_t ws = t < 8 ? s_warp[t] : 0u;
        uint32_t wi = ws;
#pragma unroll
        for (int off = 1; off < 8; off <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, wi, off);
            if (t >= off) wi += y;
        }
        if (t < 8) s_warp[t] = wi - ws;  // exclusive warp offsets
        uint32_t total = __shfl_sync(0xffffffffu, wi, 7);
        if (t == 0) {
            uint32_t excl = 0;
            uint32_t *my = tile_status + tile;
            if (tile == 0) {
                st_volatile(my, kFlagIncl | (total & kValMask));
            } else {
                st_volatile(my, kFlagAgg | (total & kValMask));
                int j = (int)tile - 1;
                uint32_t spins = 0;
                bool inject;
                const uint32_t limit = wait_limit(st, kSpinLimit, inject);
                while (j >= 0) {
                    uint32_t s = ld_volatile(tile_status + j);
                    uint32_t f = inject ? 0u : (s & ~kValMask);
                    if (f == 0u) {
                        if (++spins > limit) {
                            set_flag(st, APBF_FLAG_SPIN_LIMIT);
                            st->spin_where = 2u;
                            break;
                        }
                        __nanosleep(32);
                        continue;
                    }
                    excl += s & kValMask;
                    if (f == kFlagIncl) break;
                    --j;
                }
                st_volatile(my, kFlagIncl | ((excl + total) & kValMask));
            }
            s_excl = excl;
        }
    }
    __syncthreads();
    const uint32_t off = s_excl + s_warp[w] + (x - sum);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        uint32_t idx = base + k;
        if (idx < n) data[idx] = v[k] + off;
    }
}

}  // namespace

constexpr int kSortCarveout = 75;  // percent
apbf_status sort_prepare_device() {
    APBF_CUDA(cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSort)));
    // kernels that overlap want the same split of an SM's memory, or it drains between them
    APBF_CUDA(cudaFuncSetAttribute(k_digit_count<8>, cudaFuncAttributePreferredSharedMemoryCarveout, kSortCarveout));
    APBF_CUDA(cudaFuncSetAttribute(k_digit_scatter<8>, cudaFuncAttributePreferredSharedMemoryCarveout, kSortCarveout));
    APBF_CUDA(cudaFuncSetAttribute(k_onesweep<8>, cudaFuncAttributePreferredSharedMemoryCarveout, kSortCarveout));
    return APBF_OK;
}

static apbf_status launch_hist(apbf_ctx *ctx, const uint32_t *keys_in, const uint32_t *d_count, uint32_t max_count,
                               uint32_t key_mask, int passes, int dbits, cudaStream_t s) {
    APBF_BEFORE_LAUNCH(ctx, s, "k_sort_hist");
    const int hgrid = grid_for(ctx, max_count, 256, 4);
    if (dbits == 6)
        k_sort_hist<6><<<hgrid, 256, 0, s>>>(keys_in, d_count, max_count, key_mask, passes, ctx->sort_hist);
    else if (dbits == 7)
        k_sort_hist<7><<<hgrid, 256, 0, s>>>(keys_in, d_count, max_count, key_mask, passes, ctx->sort_hist);
    else
        k_sort_hist<8><<<hgrid, 256, 0, s>>>(keys_in, d_count, max_count, key_mask, passes, ctx->sort_hist);
    APBF_AFTER_LAUNCH(ctx, s, "k_sort_hist");
    return APBF_OK;
}

bool sort_takes_counts(const apbf_ctx *ctx, uint32_t max_count) {
    const uint32_t d = ctx->tuning.sort_digit_bits;
    return d != 6u && d != 7u && max_count > kSmallKeys && max_count <= kWaitFree;
}

// Stable sort by the low key_bits bits of the keys (rounded up to whole 4-bit
// digits exactly as the reference's pass loop, algorithms.cpp:73).  counts (may be null;
// only where sort_takes_counts): the keys' 8-bit digits already counted, passes x 256.
// behind_kernel: the keys come from a kernel just launched on s.
apbf_status sort_pairs_device(apbf_ctx *ctx, const uint32_t *keys_in, const uint32_t *vals_in, const uint32_t *d_count,
                              uint32_t max_count, uint32_t key_bits, uint32_t *keys_out, uint32_t *vals_out,
                              cudaStream_t s, const uint32_t *counts, bool behind_kernel) {
    if (max_count == 0) return APBF_OK;
    if (max_count >= (1u << 30)) return APBF_ERR_INVALID_ARG;
    uint32_t nib = (key_bits + 3u) / 4u;  // 4-bit subkeys the reference would sort
    if (nib > 8u) nib = 8u;
    uint32_t bits = nib * 4u;
    uint32_t key_mask = bits >= 32u ? 0xffffffffu : ((1u << bits) - 1u);
    const uint32_t dbits = ctx->tuning.sort_digit_bits == 6u || ctx->tuning.sort_digit_bits == 7u
                               ? ctx->tuning.sort_digit_bits
                               : 8u;  // digit width: the tuner's choice, 8 by default
    const uint32_t nb = 1u << dbits;
    int passes = (int)((bits + dbits - 1u) / dbits);
    uint32_t tiles = (max_count + kSortTile - 1) / kSortTile;
    if (tiles > ctx->sort_tiles) return APBF_ERR_INVALID_ARG;
    if (passes == 0) {
        APBF_CUDA(cudaMemcpyAsync(keys_out, keys_in, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        APBF_CUDA(cudaMemcpyAsync(vals_out, vals_in, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        return APBF_OK;
    }
    if (dbits == 8u && max_count <= kSmallKeys) {
        APBF_BEFORE_LAUNCH(ctx, s, "k_sort_small");
        APBF_CUDA(launch_behind(behind_kernel && !ctx->in_batch, k_sort_small, 1, kSmallThreads, sizeof(SmallSort), s, keys_in,
                                vals_in, keys_out, vals_out, d_count, max_count, key_mask, passes));
        APBF_AFTER_LAUNCH(ctx, s, "k_sort_small");
        return APBF_OK;
    }
    // scratch: hist passes x nb <= 4 x 256 words, status passes x tiles x nb <= 4 x tiles x 256
    // one block of memory: counters, histograms, status words or group counts (one clear)
    const bool wait_free = dbits == 8u && max_count > kWaitFree;
    const uint32_t groups = (tiles + kSortGroup - 1) / kSortGroup;
    APBF_CUDA(cudaMemsetAsync(ctx->sort_counters, 0,
                              (kSortScratchHead + (size_t)passes * (wait_free ? groups * 256u : tiles * nb)) *
                                  sizeof(uint32_t), s));
    if (!wait_free && !counts) {
        const apbf_status r = launch_hist(ctx, keys_in, d_count, max_count, key_mask, passes, (int)dbits, s);
        if (r != APBF_OK) return r;
    }
    // Ping-pong between the output (A) and scratch (B) so that the last pass lands
    // in the output: pass p writes A when (passes - 1 - p) is even.  An input that
    // aliases the output is first copied to a second scratch buffer.
    const uint32_t *src_k = keys_in, *src_v = vals_in;
    if (keys_in == keys_out || vals_in == vals_out || keys_in == vals_out || vals_in == keys_out) {
        APBF_CUDA(cudaMemcpyAsync(ctx->keys[0], keys_in, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        APBF_CUDA(cudaMemcpyAsync(ctx->vals[0], vals_in, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        src_k = ctx->keys[0];
        src_v = ctx->vals[0];
    }
    // a pass starts as the one before it ends: 12 passes over 64 019 codes 303 -> 283 us a
    // frame, 3 over 19 683 keys 211 -> 203 (not in a batch, whose waiting blocks would keep
    // other scenes' off the SMs)
    const bool behind = !ctx->in_batch;
    for (int p = 0; p < passes; ++p) {
        bool to_out = ((passes - 1 - p) & 1) == 0;
        uint32_t *dk = to_out ? keys_out : ctx->keys[1];
        uint32_t *dv = to_out ? vals_out : ctx->vals[1];
        const int sh = (int)dbits * p;
        if (wait_free) {
            uint32_t *gc = ctx->sort_status + (size_t)p * groups * 256u;  // cleared above
            uint32_t *tc = ctx->sort_status + (size_t)passes * groups * 256u;
            APBF_BEFORE_LAUNCH(ctx, s, "k_digit_count");
            APBF_CUDA(launch_behind(behind && p > 0, k_digit_count<8>, (int)tiles, kSortThreads, 0, s, src_k, d_count,
                                    max_count, key_mask, sh, tc, gc));
            APBF_AFTER_LAUNCH(ctx, s, "k_digit_count");
            APBF_BEFORE_LAUNCH(ctx, s, "k_digit_scatter");
            APBF_CUDA(launch_behind(behind, k_digit_scatter<8>, (int)tiles, kSortThreads, 0, s, src_k, src_v, dk, dv,
                                    d_count, max_count, key_mask, sh, tc, gc));
            APBF_AFTER_LAUNCH(ctx, s, "k_digit_scatter");
            src_k = dk;
            src_v = dv;
            continue;
        }
        APBF_BEFORE_LAUNCH(ctx, s, "k_onesweep");
        const uint32_t *hp = (counts ? counts : ctx->sort_hist) + p * nb;
        uint32_t *tp = ctx->sort_status + (size_t)p * tiles * nb;
        if (dbits == 6u)
            APBF_CUDA(launch_behind(behind && p > 0, k_onesweep<6>, (int)tiles, kSortThreads, 0, s, src_k, src_v, dk, dv,
                                    d_count, max_count, key_mask, sh, hp, ctx->sort_counters + p, tp, ctx->status));
        else if (dbits == 7u)
            APBF_CUDA(launch_behind(behind && p > 0, k_onesweep<7>, (int)tiles, kSortThreads, 0, s, src_k, src_v, dk, dv,
                                    d_count, max_count, key_mask, sh, hp, ctx->sort_counters + p, tp, ctx->status));
        else
            APBF_CUDA(launch_behind(behind && p > 0, k_onesweep<8>, (int)tiles, kSortThreads, 0, s, src_k, src_v, dk, dv,
                                    d_count, max_count, key_mask, sh, hp, ctx->sort_counters + p, tp, ctx->status));
        APBF_AFTER_LAUNCH(ctx, s, "k_onesweep");
        src_k = dk;
        src_v = dv;
    }
    if (src_k != keys_out) {
        APBF_CUDA(cudaMemcpyAsync(keys_out, src_k, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        APBF_CUDA(cudaMemcpyAsync(vals_out, src_v, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
    }
    return APBF_OK;
}

apbf_status prefix_sum_device(apbf_ctx *ctx, uint32_t *d_values, const uint32_t *d_count, uint32_t max_count,
                              cudaStream_t s) {
    if (max_count == 0) return APBF_OK;
    if (max_count >= (1u << 30)) return APBF_ERR_INVALID_ARG;
    uint32_t tiles = (max_count + kScanTile - 1) / kScanTile;
    if (tiles > ctx->sort_tiles * 256u) return APBF_ERR_INVALID_ARG;
    APBF_CUDA(cudaMemsetAsync(ctx->sort_counters + 7, 0, sizeof(uint32_t), s));
    APBF_CUDA(cudaMemsetAsync(ctx->sort_status, 0, (size_t)tiles * sizeof(uint32_t), s));
    APBF_BEFORE_LAUNCH(ctx, s, "k_scan");
    k_scan<<<tiles, 256, 0, s>>>(d_values, d_count, max_count, ctx->sort_counters + 7, ctx->sort_status, ctx->status);
    APBF_AFTER_LAUNCH(ctx, s, "k_scan");
    return APBF_OK;
}

}  // namespace apbf

// ---------------------------------------------------------------------------
// Allocation-free variant of the stable radix sort (apbf_sort_pairs_noalloc).
//
// Some callers cannot call cudaMalloc: a host whose device memory belongs to
// another allocator, or a per-frame path on which cudaMalloc / cudaFree would
// synchronise the device and stall the frame.  For them this entry point keeps
// its scratch (the second key/value buffer, digit histograms, tile counters and
// look-back words) in one file-scope device array of fixed size, so a call needs
// no context and allocates nothing.  Every device that loads the library holds
// the array (about 10 MB) until the process exits.
namespace apbf {
namespace {

constexpr uint32_t kNoAllocMax = 1u << 20;  // largest max_count accepted
constexpr uint32_t kNoAllocTiles = (kNoAllocMax + kSortTile - 1) / kSortTile;

struct NoAllocScratch {
    uint32_t keys[kNoAllocMax];
    uint32_t vals[kNoAllocMax];
    uint32_t hist[4 * 256];
    uint32_t counters[8];
    uint32_t tile_status[4 * kNoAllocTiles * 256];
    Status status;
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

constexpr int kMaxDevices = 64;
NoAllocScratch *g_noalloc_addr[kMaxDevices] = {};
int g_noalloc_sms[kMaxDevices] = {};
std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device (looked up once per
// device; a host-side use of g_noalloc_scratch would name host memory).
apbf_status noalloc_scratch(int dev, NoAllocScratch **out, int *sms) {
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("apbf_sort_pairs_noalloc: device ordinal out of range");
        return APBF_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_check(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        int n = 0;
        e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return cuda_check(e, "cudaDeviceGetAttribute");
        g_noalloc_addr[dev] = (NoAllocScratch *)p;
        g_noalloc_sms[dev] = n;
    }
    *out = g_noalloc_addr[dev];
    *sms = g_noalloc_sms[dev];
    return APBF_OK;
}

}  // namespace
}  // namespace apbf

extern "C" apbf_status apbf_sort_pairs_noalloc(const uint32_t *d_keys, const uint32_t *d_values,
                                               const uint32_t *d_count, uint32_t max_count,
                                               uint32_t value_upper_bound, uint32_t *d_out_keys,
                                               uint32_t *d_out_values, void *stream) {
    using namespace apbf;
    if (!d_keys || !d_values || !d_count || !d_out_keys || !d_out_values) {
        set_error("apbf_sort_pairs_noalloc: null pointer");
        return APBF_ERR_INVALID_ARG;
    }
    if (max_count > kNoAllocMax) {
        set_error("apbf_sort_pairs_noalloc: max_count above the fixed scratch size of 1048576 elements");
        return APBF_ERR_INVALID_ARG;
    }
    {  // each output range [p, p + 4 max_count) must overlap no other buffer's range
        const uintptr_t bytes = (uintptr_t)max_count * 4u;
        auto overlap = [bytes](const void *x, const void *y) {
            const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
            return bytes != 0 && a < b + bytes && b < a + bytes;
        };
        if (overlap(d_out_keys, d_out_values) || overlap(d_out_keys, d_keys) || overlap(d_out_keys, d_values) ||
            overlap(d_out_values, d_keys) || overlap(d_out_values, d_values)) {
            set_error("apbf_sort_pairs_noalloc: an output overlaps an input or the other output");
            return APBF_ERR_INVALID_ARG;
        }
    }
    if (max_count == 0) return APBF_OK;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_check(e, "cudaGetDevice");
    NoAllocScratch *sc = nullptr;
    int sms = 0;
    apbf_status r = noalloc_scratch(dev, &sc, &sms);
    if (r != APBF_OK) return r;
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t bits = 0;
    for (uint32_t v = value_upper_bound; v; v >>= 1) ++bits;
    uint32_t nib = (bits + 3u) / 4u;
    if (nib > 8u) nib = 8u;
    bits = nib * 4u;
    const uint32_t key_mask = bits >= 32u ? 0xffffffffu : ((1u << bits) - 1u);
    const int passes = (int)((bits + 7u) / 8u);
    const uint32_t tiles = (max_count + kSortTile - 1) / kSortTile;
    if (passes == 0) {
        APBF_CUDA(cudaMemcpyAsync(d_out_keys, d_keys, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        APBF_CUDA(cudaMemcpyAsync(d_out_values, d_values, (size_t)max_count * 4, cudaMemcpyDeviceToDevice, s));
        return APBF_OK;
    }
    // the array keeps the previous call's contents: clear what must start at zero
    APBF_CUDA(cudaMemsetAsync(sc->hist, 0, sizeof(sc->hist), s));
    APBF_CUDA(cudaMemsetAsync(sc->counters, 0, sizeof(sc->counters), s));
    APBF_CUDA(cudaMemsetAsync(sc->tile_status, 0, (size_t)passes * tiles * 256 * sizeof(uint32_t), s));
    APBF_CUDA(cudaMemsetAsync(&sc->status, 0, sizeof(Status), s));
    uint64_t need = ((uint64_t)max_count + 255) / 256;
    const int hist_grid = (int)std::min<uint64_t>(std::max<uint64_t>(need, 1), (uint64_t)sms * 4);
    k_sort_hist<8><<<hist_grid, 256, 0, s>>>(d_keys, d_count, max_count, key_mask, passes, sc->hist);
    APBF_CUDA(cudaGetLastError());
    const uint32_t *src_k = d_keys, *src_v = d_values;
    for (int p = 0; p < passes; ++p) {
        const bool to_out = ((passes - 1 - p) & 1) == 0;
        uint32_t *dk = to_out ? d_out_keys : sc->keys;
        uint32_t *dv = to_out ? d_out_values : sc->vals;
        k_onesweep<8><<<tiles, kSortThreads, 0, s>>>(src_k, src_v, dk, dv, d_count, max_count, key_mask, 8 * p,
                                         sc->hist + p * 256, sc->counters + p,
                                         sc->tile_status + (size_t)p * tiles * 256, &sc->status);
        APBF_CUDA(cudaGetLastError());
        src_k = dk;
        src_v = dv;
    }
    return APBF_OK;
}
