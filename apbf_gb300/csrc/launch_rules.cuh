// launch_rules.cuh -- rules that pick launch shapes and places from sizes and settings.  Plain
// C++, so that a host test can go through them without a device.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define APBF_RULE __host__ __device__ __forceinline__
#else
#define APBF_RULE inline
#endif

namespace apbf {

// Threads per particle, threads per block and blocks per SM (at most) of the direct Jacobi passes.
struct PassShape {
    uint32_t lanes, block, per_sm;
};
// The shape fields of a context's apbf_tuning at creation.  They stand for the automatic
// shape, so a tuning that changes other fields only, or writes back what apbf_get_tuning
// returned, leaves the choice where it was.
constexpr PassShape kAutomaticShape = {1u, 256u, 8u};

APBF_RULE PassShape pass_shape_rule(PassShape tuned, uint32_t capacity, bool features) {
    PassShape sh = tuned;
    const bool automatic = tuned.lanes == kAutomaticShape.lanes && tuned.block == kAutomaticShape.block &&
                           tuned.per_sm == kAutomaticShape.per_sm;
    if (automatic) {
        // Several threads share a row while the particles alone leave the chip's schedulers
        // short of warps: a frame of 2 197 particles takes 325 / 299 / 279 us with 1 / 2 / 4
        // threads, 32 768 particles 2107 / 1742 / 1756, 64 019 506 / 501 / 520, 119 771
        // 2625 / 2751 / 3227.
        sh.lanes = capacity > 98304u ? 1u : capacity > 32768u ? 2u : 4u;
        sh.per_sm = 32u;  // a thread per particle and lane
    }
    // The features' float sums keep the row's order: one thread per particle under any shape,
    // or the applied lambda of a learned pass would depend on the tuning.
    if (features) sh.lanes = 1u;
    // One thread per particle: blocks that are all resident and take several particles per
    // thread, as every block begins with the sums of the pass before it.  Density and position
    // pass at 262 144 particles 75.8 us with blocks of 256, a particle per thread, 73.1 so; at
    // a million 250.5 and 234.4, with 6 neighbours instead of 32 102.1 and 85.7.
    if (automatic && sh.lanes == 1u) {
        sh.block = 128u;
        sh.per_sm = 8u;
    }
    return sh;
}

// Particles of a tile of the tiled passes, one thread each, or 64 with two threads each where
// 128 would leave SMs without a tile (2 197 particles: 294 us a frame with 128 x 1, 285 with
// 64 x 2; from 30 000 particles on the larger tile is as fast or faster: 1521 / 1509 us at
// 32 768, 2094 / 2570 at 119 771).
APBF_RULE uint32_t tile_particles(uint32_t capacity) { return capacity <= 24576u ? 64u : 128u; }

// Where a run of m entries starts in a pool of `size`, `before` entries having been asked of it
// (kNoRun: it does not fit).  Rows that do not fit are counted too, and a list can hold more
// than 2^32 entries: 64 bits, so that the count never comes round to places given away.
using PoolCount = unsigned long long;
constexpr uint32_t kNoRun = 0xffffffffu;
APBF_RULE uint32_t pool_run(PoolCount before, uint32_t m, uint32_t size) {
    return before <= size && m <= size - (uint32_t)before ? (uint32_t)before : kNoRun;
}

}  // namespace apbf
