// rowwalk.cuh -- groups of threads that walk the particles around one particle and write
// its neighbour row (neighborhood.cu, neighborhood_bs.cu).
#pragma once

#include <type_traits>

#include "apbf_internal.cuh"

namespace apbf {

constexpr uint32_t kBuildThreads = 256, kRowStage = 64;

// Squared distance of two fixed-point positions when no axis differs by more than R
// (else ~0: the pair is beyond R whatever the other axes).  FAST: their differences stay
// below 2^31 (both lie inside a grid of that size), so three squares cannot overflow the
// sum and no range test is needed.
template <bool FAST>
__device__ __forceinline__ unsigned long long dist2_within(int4 a, int4 b, uint32_t R) {
    if (FAST) {
        const long long dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
        return (unsigned long long)(dx * dx) + (unsigned long long)(dy * dy) + (unsigned long long)(dz * dz);
    }
    long long dx = (long long)b.x - a.x, dy = (long long)b.y - a.y, dz = (long long)b.z - a.z;
    dx = dx < 0 ? -dx : dx;
    dy = dy < 0 ? -dy : dy;
    dz = dz < 0 ? -dz : dz;
    if (dx > (long long)R || dy > (long long)R || dz > (long long)R) return ~0ull;
    const uint32_t ax = (uint32_t)dx, ay = (uint32_t)dy, az = (uint32_t)dz;
    return (unsigned long long)ax * ax + (unsigned long long)ay * ay + (unsigned long long)az * az;
}

// Sum over a group of G consecutive lanes.
template <int G>
__device__ __forceinline__ uint32_t group_total(uint32_t v) {
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

// The row of particle i as a group of G threads builds it.  Each thread brings a run
// [s, s + len) of the list; `take` joins the group's runs in thread order and tests G
// candidates at a time against |x_j - x_i| <= R, whatever run they come from.  A ballot
// gives the kept ones their places, so the row keeps the runs' order.  Rows are collected
// in shared memory (s_row, kRowStage entries; the rest goes out directly) and written by
// `write_rows` a line at a time, as they are read later.  Every lane of the warp calls
// these together.
template <int G>
struct RowWalk {
    static constexpr uint32_t kParticles = kBuildThreads / G;  // per block
    static constexpr uint32_t kPad = kParticles + 1;           // a group's next places fall into other banks
    const int4 *rec;  // the list's positions (w: search radius, read when radii are compared)
    uint32_t *idx;
    uint32_t stride, maxn;
    uint32_t *s_row;
    uint32_t i, gl, slot, shift, below, mine;
    int4 p;
    uint32_t R;
    unsigned long long R2;
    bool radii;                      // count the one-sided pairs
    uint32_t count = 0, one_sided = 0;

    __device__ __forceinline__ RowWalk(const int4 *rec_, uint32_t *idx_, uint32_t stride_, uint32_t maxn_, uint32_t *s_row_,
                                       bool radii_)
        : rec(rec_), idx(idx_), stride(stride_), maxn(maxn_), s_row(s_row_), radii(radii_) {
        gl = threadIdx.x % G;
        slot = threadIdx.x / G;
        shift = threadIdx.x & 31u & ~(uint32_t)(G - 1);  // the group's first lane in its warp
        below = (1u << gl) - 1u;
        mine = G == 32 ? 0xffffffffu : (1u << G) - 1u;
    }
    __device__ __forceinline__ void start(uint32_t i_, int4 p_, uint32_t R_) {
        i = i_;
        p = p_;
        R = R_;
        R2 = (unsigned long long)R_ * R_;
        count = one_sided = 0;
    }
    template <bool FAST>
    __device__ __forceinline__ void test(bool in, uint32_t j, int4 q) {
        const unsigned long long d2 = dist2_within<FAST>(p, q, R);
        const bool keep = in && j != i && d2 <= R2;
        const uint32_t bal = (__ballot_sync(0xffffffffu, keep) >> shift) & mine;
        if (keep) {
            const uint32_t at = count + __popc(bal & below);
            if (at < kRowStage) s_row[at * kPad + slot] = j;
            else if (at < maxn) idx[(size_t)at * stride + i] = j;
            if (radii) {
                const unsigned long long Rj = (unsigned long long)(uint32_t)max(q.w, 0);
                one_sided += (q.w >= 0 && d2 <= Rj * Rj) ? 0u : 1u;
            }
        }
        count += __popc(bal);
    }
    template <bool FAST>
    __device__ __forceinline__ void take(uint32_t s, uint32_t len) {
        uint32_t incl = len;
#pragma unroll
        for (int off = 1; off < G; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, off, G);
            if ((int)gl >= off) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, G - 1, G);
        const uint32_t adj = s - (incl - len);  // candidate f of the joined runs is particle adj + f
        const uint32_t rounds = __reduce_max_sync(0xffffffffu, total);
        const auto candidate = [&](uint32_t f) {  // of the thread whose run holds f
            uint32_t k = 0;
#pragma unroll
            for (int off = G / 2; off > 0; off >>= 1)
                if (__shfl_sync(0xffffffffu, incl, k + off - 1, G) <= f) k += off;
            return __shfl_sync(0xffffffffu, adj, k, G) + f;
        };
        for (uint32_t w = 0; w < rounds; w += 2 * G) {  // two candidates of each thread in flight
            const uint32_t f0 = w + gl, f1 = f0 + G, j0 = candidate(f0);
            const bool in0 = f0 < total, in1 = f1 < total;
            const int4 q0 = in0 ? rec[j0] : p;
            if (w + G < rounds) {
                const uint32_t j1 = candidate(f1);
                const int4 q1 = in1 ? rec[j1] : p;
                test<FAST>(in0, j0, q0);
                test<FAST>(in1, j1, q1);
            } else {  // (of short runs, as sparse lists have, the last round holds one)
                test<FAST>(in0, j0, q0);
            }
        }
    }
    // The block's rows, entries [0, s_cnt[slot]) of each (after a barrier behind the walks).
    __device__ __forceinline__ void write_rows(const uint32_t *s_cnt, uint32_t base) const {
        const uint32_t pl = threadIdx.x % kParticles, m = min(s_cnt[pl], kRowStage);
        for (uint32_t k = threadIdx.x / kParticles; k < m; k += kBuildThreads / kParticles)
            idx[(size_t)k * stride + base + pl] = s_row[k * kPad + pl];
    }
};

// Adds a block's kept pairs to the total: one addition per block, since a word that many SMs
// write costs about 25 ns a time.  Every thread of the block calls it.
__device__ __forceinline__ void add_pairs(unsigned long long *total, unsigned long long local) {
    __shared__ unsigned long long s_local;
    if (threadIdx.x == 0) s_local = 0ull;
    __syncthreads();
    for (int off = 16; off > 0; off >>= 1) local += __shfl_down_sync(0xffffffffu, local, off);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(&s_local, local);
    __syncthreads();
    if (threadIdx.x == 0 && s_local) atomicAdd(total, s_local);
}

// box_push as a call: it runs once per particle, and the walks are bound by their
// instructions.
__device__ __noinline__ static int4 box_push_call(int4 ip, float r, uint32_t id, const float4 *__restrict__ bmin,
                                           const float4 *__restrict__ bmax, const float4 *__restrict__ rot,
                                           uint32_t nb) {
    return box_push(ip, r, id, bmin, bmax, rot, nb);
}

}  // namespace apbf
