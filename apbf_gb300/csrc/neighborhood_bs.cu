// neighborhood_bs.cu -- neighborhood_binary_search::apply
// (source/neighborhood_binary_search.cpp:22-75), the reference's default search
// (shaders/cpu_gpu_shared_config.h:5).
//
//  1. k_code_word + sort_pairs_device, three times: stable sort of the particles by
//     the 96-bit interleave of their raw coordinates, least significant 32-bit word
//     first, so that ties keep the list order (neighborhood_binary_search.cpp:43-47,
//     calculate_position_code.comp:22-72).
//  2. reorder_particles: gather every attribute, remap the transfer and glue lists
//     (neighborhood_binary_search.cpp:49-50).
//  3. k_sorted_codes: the codes of the sorted particles (:52-56), and the cells of their
//     radii's level into a hash table.
//  4. k_bs_rows: per particle, the 27 cells of edge 2^k around its own cell; each
//     cell's particles are one run of the sorted codes, found in the table when all radii
//     have one level, else by two searches (neighborhood_binary_search.comp:186-275).
//
// Canonical rules where the reference's arithmetic is not exact:
//  * the level k is the smallest with 2^k >= R, R the canonical fixed-point search
//    radius floor(kw * scale * 2^18) of the Green search, instead of
//    ceil(log2(range * 2^18)) in FP32 (comp:188): exact, and still cells at least R
//    wide, so the 27 cells hold every particle within R;
//  * the neighbour predicate is the Green search's exact integer one,
//    |x_j - x_i|^2 <= R^2, instead of an FP32 distance (comp:271);
//  * the lower bound is searched over the whole sorted list: the reference's
//    block-local shortcut (comp:104-108) can start inside a run of equal codes
//    that begins in an earlier block;
//  * at k = 31 each axis has two cells, so the offsets -1 and +1 name the same cell;
//    it is scanned once (the reference scans it twice and lists those neighbours
//    twice).
#include "rowwalk.cuh"

namespace apbf {
namespace {

// Bits 0..20 of v moved to bits 0, 3, 6, ..., 60.
__device__ __forceinline__ unsigned long long spread21(uint32_t v) {
    unsigned long long x = v & 0x1fffffu;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

// Code bit 3b + a is bit b of axis a (x = 0, y = 1, z = 2), the coordinates taken as
// uint32 (calculate_position_code.comp:22-62).  .x holds code bits 0-63, .y bits 64-95.
__device__ __forceinline__ ulonglong2 code96(uint32_t x, uint32_t y, uint32_t z) {
    const unsigned long long lo = spread21(x) | spread21(y) << 1 | spread21(z) << 2;
    const unsigned long long t = spread21(x >> 21) | spread21(y >> 21) << 1 | spread21(z >> 21) << 2;
    return make_ulonglong2(lo | t << 63, t >> 1);
}

__device__ __forceinline__ bool less96(ulonglong2 a, ulonglong2 b) {
    return a.y < b.y || (a.y == b.y && a.x < b.x);
}

__device__ __forceinline__ uint32_t code_word(ulonglong2 c, uint32_t w) {
    return w == 0 ? (uint32_t)c.x : (w == 1 ? (uint32_t)(c.x >> 32) : (uint32_t)c.y);
}

// keys[k] = word w of the code of particle o, vals[k] = o, with o = order[k] (k when
// order is null).
__global__ void k_code_word(const int4 *__restrict__ pos, const uint32_t *d_len, uint32_t w,
                            const uint32_t *__restrict__ order, uint32_t *__restrict__ keys,
                            uint32_t *__restrict__ vals) {
    const uint32_t n = d_len[kLenParticles];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t o = order ? order[k] : k;
        const int4 p = pos[o];
        keys[k] = code_word(code96((uint32_t)p.x, (uint32_t)p.y, (uint32_t)p.z), w);
        if (vals) vals[k] = o;
    }
}

// Word 0 of every particle's code, and the counts of all twelve 8-bit digits of the codes
// (counts: 12 x 256, cleared): how often a digit occurs does not depend on the order, so the
// three sorts need no pass over their keys for it (three launches of 4 us each).
__global__ void __launch_bounds__(512) k_code_counts(const int4 *__restrict__ pos, const uint32_t *d_len,
                                                     uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                                                     uint32_t *__restrict__ counts) {
    __shared__ uint32_t sh[12 * 256];
    for (uint32_t q = threadIdx.x; q < 12u * 256u; q += blockDim.x) sh[q] = 0u;
    __syncthreads();
    const uint32_t n = d_len[kLenParticles];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int4 p = pos[k];
        const ulonglong2 c = code96((uint32_t)p.x, (uint32_t)p.y, (uint32_t)p.z);
        keys[k] = code_word(c, 0);
        vals[k] = k;
#pragma unroll
        for (int d = 0; d < 12; ++d)
            atomicAdd(&sh[d * 256 + (int)((code_word(c, d / 4) >> (8 * (d % 4))) & 255u)], 1u);
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < 12u * 256u; q += blockDim.x)
        if (sh[q]) atomicAdd(&counts[q], sh[q]);
}

// The cells of one level as a hash table: 63-bit cell number + 1 (0: empty), first particle
// and end of the cell's run of the sorted list.
struct __align__(16) BsCell {
    unsigned long long key;
    uint32_t start, end;
};
__device__ __forceinline__ unsigned long long bs_key(uint32_t ux, uint32_t uy, uint32_t uz) {
    return 1ull + ((unsigned long long)ux | (unsigned long long)uy << 21 | (unsigned long long)uz << 42);
}
__device__ __forceinline__ uint32_t bs_hash(unsigned long long key, uint32_t mask) {
    return (uint32_t)((key * 0x9E3779B97F4A7C15ull) >> 32) & mask;
}
// The level of a search radius: the smallest k with 2^k >= R (R < 2^31, so k <= 31).
__device__ __forceinline__ uint32_t bs_level(long long R) {
    return R <= 1 ? 0u : 32u - (uint32_t)__clz((uint32_t)(R - 1));
}
constexpr uint32_t kTableLevel = 11;  // from this level on a cell number has at most 63 bits

// Also: the transfer list follows the reorder, the first thread resets what the search
// and the solve behind it count from, and the particles enter the cells of their radius's
// level into the table (the first of a cell's run its start, the last its end).  The table
// holds every cell when all radii have one level; the levels' range tells: 32 less the
// lowest, and the highest.  (table and levels cleared beforehand.)
__global__ void k_sorted_codes(const int4 *pos, const float *width, float scale, const uint32_t *d_len,
                               ulonglong2 *code, BsCell *table, uint32_t mask, uint32_t *levels, TransferBufs tr,
                               const uint32_t *inv_perm, Status *st, unsigned long long *total) {
    grid_dependency_wait();
    grid_dependency_trigger();
    const uint32_t n = d_len[kLenParticles];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_search(st, total);
    remap_transfers(tr, inv_perm, d_len, st);
    uint32_t low = 0u, high = 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int4 p = pos[i];
        code[i] = code96((uint32_t)p.x, (uint32_t)p.y, (uint32_t)p.z);
        const long long R = range_fixed(width[i], scale);
        if (R < 0) {  // no cell of its own, but it may open or close another's run
            low = 32u;
            continue;
        }
        const uint32_t k = bs_level(R);
        low = max(low, 32u - k);
        high = max(high, k);
        if (k < kTableLevel || !table) continue;
        const uint32_t ux = (uint32_t)p.x >> k, uy = (uint32_t)p.y >> k, uz = (uint32_t)p.z >> k;
        const auto same = [&](int4 q) {
            return (uint32_t)q.x >> k == ux && (uint32_t)q.y >> k == uy && (uint32_t)q.z >> k == uz;
        };
        const bool opens = i == 0u || !same(pos[i - 1u]), closes = i + 1u == n || !same(pos[i + 1u]);
        if (!opens && !closes) continue;
        const unsigned long long key = bs_key(ux, uy, uz);
        for (uint32_t h = bs_hash(key, mask);; h = (h + 1u) & mask) {  // (never full: more slots than particles)
            const unsigned long long was = atomicCAS(&table[h].key, 0ull, key);
            if (was != 0ull && was != key) continue;
            if (opens) table[h].start = i;
            if (closes) table[h].end = i + 1u;
            break;
        }
    }
    low = __reduce_max_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    if ((threadIdx.x & 31u) == 0u) {  // (a bound that already holds is left alone)
        if (low > *(volatile uint32_t *)&levels[0]) atomicMax(&levels[0], low);
        if (high > *(volatile uint32_t *)&levels[1]) atomicMax(&levels[1], high);
    }
}

// First index j in [0, n) with !before(code[j]) (n when none), for a predicate that holds
// for a prefix of the list; searched outward from `hint` with doubling steps and then
// bisected: cells near a particle are mostly near it in the sorted order.
template <typename F>
__device__ __forceinline__ uint32_t first_not(const ulonglong2 *code, uint32_t n, uint32_t hint, F before) {
    uint32_t lo, hi;  // the answer lies in [lo, hi]
    if (before(code[hint])) {
        uint32_t a = hint, step = 1;  // before(code[a])
        for (;;) {
            const uint32_t b = step <= n - 1 - a ? a + step : n;  // index to probe, or n
            if (b >= n) {
                lo = a + 1;
                hi = n;
                break;
            }
            if (!before(code[b])) {
                lo = a + 1;
                hi = b;
                break;
            }
            a = b;
            step <<= 1;
        }
    } else {
        uint32_t b = hint, step = 1;  // !before(code[b])
        for (;;) {
            if (b == 0) {
                lo = hi = 0;
                break;
            }
            const uint32_t a = b > step ? b - step : 0;
            if (before(code[a])) {
                lo = a + 1;
                hi = b;
                break;
            }
            b = a;
            step <<= 1;
        }
    }
    while (lo < hi) {  // bisect: hi == n or !before(code[hi]), before(code[lo - 1])
        const uint32_t mid = lo + (hi - lo) / 2;
        if (before(code[mid]))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

struct BsArgs {
    const int4 *pos;
    int4 *pos_box;  // when non-null: receives box_collision(pos) (the first Jacobi iteration's box pass)
    const ulonglong2 *code;
    const float *range;
    const float *radius;
    const float4 *bmin, *bmax, *rot;
    uint32_t nboxes;
    float scale;
    const uint32_t *d_len;
    uint32_t stride, maxn;
    uint32_t *count, *idx;
    unsigned long long *total;
    Status *st;
    const BsCell *table;  // k_sorted_codes' cells, mask + 1 slots; null: no table
    uint32_t mask;
    const uint32_t *levels;
};

// neighborhood_binary_search.comp:180-275 by groups of G threads (RowWalk): a thread per
// cell finds its run, in the table of cells when all radii have one level, else by two
// searches of the sorted codes.  The searches are about 40 dependent loads for each of 27
// cells: 178 us at 64 019 particles, with the table 55.
template <int G>
__global__ void __launch_bounds__(kBuildThreads) k_bs_rows(BsArgs a) {
    using Walk = RowWalk<G>;
    __shared__ uint32_t s_row[kRowStage * Walk::kPad];
    __shared__ uint32_t s_cnt[Walk::kParticles];
    grid_dependency_wait();
    grid_dependency_trigger();
    const uint32_t n = a.d_len[kLenParticles];
    const bool tabled = a.table && 32u - a.levels[0] == a.levels[1] && a.levels[1] >= kTableLevel;
    Walk w(a.pos, a.idx, a.stride, a.maxn, s_row, false);
    const uint32_t gl = w.gl;
    unsigned long long local = 0;
    long long rmin = 0x7fffffffffffffffll, rmax = -1;
    for (uint32_t base = blockIdx.x * Walk::kParticles; base < n; base += gridDim.x * Walk::kParticles) {
        const uint32_t i = base + w.slot;
        const bool valid = i < n;
        const int4 p = valid ? a.pos[i] : make_int4(0, 0, 0, 0);
        const long long R = valid ? range_fixed(a.range[i], a.scale) : -1;
        if (valid && R < 0 && gl == 0u) set_flag(a.st, APBF_FLAG_NONFINITE);  // NaN or negative width: no neighbours
        if (R >= 0) {
            rmin = R < rmin ? R : rmin;
            rmax = R > rmax ? R : rmax;
        }
        const uint32_t k = bs_level(R);
        const uint32_t m = k == 31 ? 2u : 3u;  // at k = 31 the offset +1 is the offset -1
        const uint32_t ncell = R < 0 ? 0u : m * m * m;
        const uint32_t ux = (uint32_t)p.x >> k, uy = (uint32_t)p.y >> k, uz = (uint32_t)p.z >> k;
        w.start(i, p, (uint32_t)(R < 0 ? 0 : R));
        const auto range = [&](uint32_t c, uint32_t &s, uint32_t &len) {  // of the c-th cell
            s = len = 0u;
            if (c >= ncell) return;
            const uint32_t t = c / m, dx = c - t * m, dz = t / m, dy = t - dz * m;
            // the cell, wrapping modulo 2^32 like the code arithmetic
            const uint32_t cx = (ux + dx - 1u) << k, cy = (uy + dy - 1u) << k, cz = (uz + dz - 1u) << k;
            if (tabled) {
                const unsigned long long key = bs_key(cx >> k, cy >> k, cz >> k);
                for (uint32_t h = bs_hash(key, a.mask);; h = (h + 1u) & a.mask) {
                    const uint4 e = *reinterpret_cast<const uint4 *>(&a.table[h]);
                    const unsigned long long found = (unsigned long long)e.y << 32 | e.x;
                    if (found == 0ull) return;
                    if (found != key) continue;
                    s = e.z;
                    len = e.w - e.z;
                    return;
                }
            }
            const uint32_t d3 = 3u * k;  // the code bits below the cell
            const ulonglong2 m96 = make_ulonglong2(d3 >= 64 ? ~0ull : (1ull << d3) - 1ull,
                                                   d3 > 64 ? (1ull << (d3 - 64)) - 1ull : 0ull);
            const ulonglong2 first = code96(cx, cy, cz);
            const ulonglong2 last = make_ulonglong2(first.x | m96.x, first.y | m96.y);
            s = first_not(a.code, n, i, [&](ulonglong2 x) { return less96(x, first); });
            if (s < n) len = first_not(a.code, n, s, [&](ulonglong2 x) { return !less96(last, x); }) - s;
        };
        uint32_t s, len;
        range(gl, s, len);
        for (uint32_t c0 = 0; c0 < 27u; c0 += G) {
            uint32_t ns, nlen;
            range(c0 + G + gl, ns, nlen);  // in flight while this round's candidates are tested
            __syncwarp();
            w.template take<false>(s, len);
            s = ns;
            len = nlen;
        }
        if (gl == 0u) {
            const uint32_t kept = min(w.count, a.maxn);
            s_cnt[w.slot] = kept;
            if (valid) {
                if (w.count > a.maxn) {
                    set_flag(a.st, APBF_FLAG_NEIGHBOR_OVERFLOW);
                    atomicMax(&a.st->required_neighbors, w.count);
                }
                a.count[i] = kept;
                local += kept;
            }
        }
        __syncthreads();
        w.write_rows(s_cnt, base);
        if (a.pos_box && threadIdx.x < Walk::kParticles && base + threadIdx.x < n) {
            const uint32_t j = base + threadIdx.x;
            a.pos_box[j] = box_push_call(a.pos[j], a.radius[j], j, a.bmin, a.bmax, a.rot, a.nboxes);
        }
        __syncthreads();  // the rows are the next particles'
    }
    add_pairs(a.total, local);
    // (a bound that already holds is left alone)
    if (gl == 0u && rmax >= 0) {
        if ((unsigned long long)rmin < *(volatile unsigned long long *)&a.st->range_min)
            atomicMin(&a.st->range_min, (unsigned long long)rmin);
        if ((unsigned long long)rmax > *(volatile unsigned long long *)&a.st->range_max)
            atomicMax(&a.st->range_max, (unsigned long long)rmax);
    }
}

}  // namespace

apbf_status neighborhood_binary_search(apbf_ctx *ctx, float range_scale, cudaStream_t s, bool fuse_box) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    const int g = grid_for(ctx, cap);
    // three stable passes, least significant word first
    // the table and the levels' range, cleared ahead, so that from the sort on
    // kernel follows kernel and each starts as the one before it ends
    BsCell *table = reinterpret_cast<BsCell *>(ctx->bs_table);
    uint32_t *levels = ctx->bs_levels;
    const bool behind = !ctx->in_batch;
    if (table) APBF_CUDA(cudaMemsetAsync(table, 0, (size_t)ctx->bs_slots * sizeof(BsCell), s));
    APBF_CUDA(cudaMemsetAsync(levels, 0, 2 * sizeof(uint32_t), s));
    const bool counted = sort_takes_counts(ctx, cap);
    if (counted) APBF_CUDA(cudaMemsetAsync(ctx->bs_counts, 0, 12 * 256 * sizeof(uint32_t), s));
    for (uint32_t w = 0; w < 3; ++w) {
        const FluidBufs &cur = ctx->fl[ctx->fcur];
        if (counted && w == 0) {
            APBF_BEFORE_LAUNCH(ctx, s, "k_code_counts");
            k_code_counts<<<grid_for(ctx, cap, 512, 2), 512, 0, s>>>(cur.pos, ctx->d_len, ctx->keys[0], ctx->vals[0],
                                                                     ctx->bs_counts);
            APBF_AFTER_LAUNCH(ctx, s, "k_code_counts");
        } else {
            APBF_BEFORE_LAUNCH(ctx, s, "k_code_word");
            k_code_word<<<g, kBlock, 0, s>>>(cur.pos, ctx->d_len, w, w ? ctx->perm : nullptr, ctx->keys[0],
                                             ctx->vals[0]);
            APBF_AFTER_LAUNCH(ctx, s, "k_code_word");
        }
        apbf_status r = sort_pairs_device(ctx, ctx->keys[0], ctx->vals[0], ctx->d_len + kLenParticles, cap, 32u,
                                          ctx->sorted_keys, ctx->perm, s,
                                          counted ? ctx->bs_counts + w * 4 * 256 : nullptr);
        if (r != APBF_OK) return r;
    }
    apbf_status r = reorder_particles(ctx, s, false, 0.0f, behind);
    if (r != APBF_OK) return r;
    FluidBufs &f = ctx->fl[ctx->fcur];
    APBF_BEFORE_LAUNCH(ctx, s, "k_sorted_codes");
    APBF_CUDA(launch_behind(behind, k_sorted_codes, g, kBlock, 0, s, f.pos, f.kernel_width, range_scale, ctx->d_len,
                            ctx->pos_code, table, ctx->bs_slots - 1u, levels, ctx->tr[ctx->tcur], ctx->inv_perm,
                            ctx->status, ctx->d_pairs));
    APBF_AFTER_LAUNCH(ctx, s, "k_sorted_codes");
    FluidBufs &spare = ctx->fl[ctx->fcur ^ 1];
    BsArgs a;
    a.pos = f.pos;
    a.pos_box = fuse_box ? spare.pos : nullptr;
    a.code = ctx->pos_code;
    a.range = f.kernel_width;
    a.radius = f.radius;
    a.bmin = ctx->box_min;
    a.bmax = ctx->box_max;
    a.rot = ctx->box_rot;
    a.nboxes = ctx->n_boxes;
    a.scale = range_scale;
    a.d_len = ctx->d_len;
    a.stride = ctx->row_stride;
    a.maxn = ctx->cfg.max_neighbors;
    a.count = ctx->nb_count;
    a.idx = ctx->nb_idx;
    a.total = ctx->d_pairs;
    a.st = ctx->status;
    a.table = table;
    a.mask = ctx->bs_slots - 1u;
    a.levels = levels;
    APBF_BEFORE_LAUNCH(ctx, s, "k_bs_rows");
    // threads per particle as in the Green search: 8 / 16 / 32 take 56 / 66 / 93 us at 64 019
    if (cap <= 12288u)
        APBF_CUDA(launch_behind(behind, k_bs_rows<32>, grid_for(ctx, cap, RowWalk<32>::kParticles, 64), kBuildThreads, 0, s, a));
    else if (cap <= 32768u)
        APBF_CUDA(launch_behind(behind, k_bs_rows<16>, grid_for(ctx, cap, RowWalk<16>::kParticles, 64), kBuildThreads, 0, s, a));
    else
        APBF_CUDA(launch_behind(behind, k_bs_rows<8>, grid_for(ctx, cap, RowWalk<8>::kParticles, 64), kBuildThreads, 0, s, a));
    APBF_AFTER_LAUNCH(ctx, s, "k_bs_rows");
    if (fuse_box) {  // the box-collided positions are the current ones now
        int4 *t = f.pos;
        f.pos = spare.pos;
        spare.pos = t;
    }
    return build_reverse_rows(ctx, s);
}

}  // namespace apbf

using namespace apbf;

extern "C" {

apbf_status apbf_neighborhood_binary_search_apply(apbf_ctx *ctx, float range_scale, void *stream) {
    if (!ctx) return APBF_ERR_INVALID_ARG;
    if (!ctx->bs_table) {  // (nothing is made while the stream is captured)
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        APBF_CUDA(cudaStreamIsCapturing((cudaStream_t)stream, &st));
        if (st == cudaStreamCaptureStatusNone) make_cell_table(ctx);
    }
    APBF_BOUND_LENGTHS(ctx, (cudaStream_t)stream);
    return neighborhood_binary_search(ctx, range_scale, (cudaStream_t)stream);
}

apbf_status apbf_calculate_position_code(apbf_ctx *ctx, const uint32_t *d_index_list, uint32_t code_section,
                                         uint32_t *d_out, void *stream) {
    if (!ctx || !d_out || code_section > 2) {
        set_error("calculate_position_code: needs an output and a code section in 0..2");
        return APBF_ERR_INVALID_ARG;
    }
    cudaStream_t s = (cudaStream_t)stream;
    APBF_BOUND_LENGTHS(ctx, s);
    const FluidBufs &f = ctx->fl[ctx->fcur];
    APBF_BEFORE_LAUNCH(ctx, s, "k_code_word");
    k_code_word<<<grid_for(ctx, ctx->cfg.particle_capacity), kBlock, 0, s>>>(f.pos, ctx->d_len, code_section,
                                                                              d_index_list, d_out, nullptr);
    APBF_AFTER_LAUNCH(ctx, s, "k_code_word");
    return APBF_OK;
}

apbf_status apbf_set_neighborhood_search(apbf_ctx *ctx, int method) {
    if (!ctx) return APBF_ERR_INVALID_ARG;
    if (method != APBF_NEIGHBORHOOD_GREEN && method != APBF_NEIGHBORHOOD_BINARY_SEARCH) {
        set_error("set_neighborhood_search: the method is APBF_NEIGHBORHOOD_GREEN or APBF_NEIGHBORHOOD_BINARY_SEARCH");
        return APBF_ERR_INVALID_ARG;
    }
    if (method != ctx->search_method) ctx->graph_version++;  // captured substeps hold the search
    ctx->search_method = method;
    if (method == APBF_NEIGHBORHOOD_BINARY_SEARCH) make_cell_table(ctx);
    make_tile_plans(ctx);
    return APBF_OK;
}

}  // extern "C"
