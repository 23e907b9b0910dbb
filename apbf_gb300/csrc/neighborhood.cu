// neighborhood.cu -- neighborhood_green::apply (source/neighborhood_green.cpp:27-77).
//
//  1. k_position_keys: Morton key of each particle's grid cell
//     (calculate_position_hash.comp:23-46; canonical integer cell mapping).
//  2. sort_pairs_device: stable sort of (key, particle id).
//  3. k_reorder: gather every particle attribute into the alternate buffer set and
//     swap (hidden_list().apply_edit + mParticles->sort(), neighborhood_green.cpp:54-56),
//     remap the transfer list (indexed_list.h:288-308).
//  4. k_cell_ranges: [start, end) of every occupied cell (find_value_ranges.comp).
//  5. k_build_rows: per particle, walk the cells overlapping [X - R, X + R] and keep
//     every other particle within R (neighborhood_green.comp:49-87), written
//     column-major so that consecutive particles' k-th entries are contiguous.
//     When the search radii differ it also writes correction rows into the
//     reverse-row arrays (the rare one-sided pairs), so that the position-update
//     pass gathers over the particle's own row plus its corrections instead of
//     scattering with atomics, and no transpose is needed.
//  6. k_reverse_rows (binary-search rows and pruned rows): the transpose.
#include <algorithm>

#include "apbf_internal.cuh"
#include "rowwalk.cuh"

namespace apbf {
namespace {

struct Bounds {
    long long lo[3];
    long long hi[3];
};

Bounds fixed_bounds(const float minp[3], const float maxp[3]) {
    Bounds b;
    for (int d = 0; d < 3; ++d) {
        b.lo[d] = llround((double)minp[d] * 262144.0);
        b.hi[d] = llround((double)maxp[d] * 262144.0);
        if (b.hi[d] <= b.lo[d]) b.hi[d] = b.lo[d] + 1;
    }
    return b;
}

// Its first thread also resets what the search and the solve behind it count from.
__global__ void k_position_keys(const int4 *__restrict__ pos, const uint32_t *d_len, Bounds b, uint32_t L,
                                uint32_t *__restrict__ keys, uint32_t *__restrict__ seq, Status *st,
                                unsigned long long *total) {
    uint32_t n = d_len[kLenParticles];
    if (blockIdx.x == 0 && threadIdx.x == 0) reset_search(st, total);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int4 p = pos[i];
        uint32_t cx = cell_coord(p.x, b.lo[0], b.hi[0], L);
        uint32_t cy = cell_coord(p.y, b.lo[1], b.hi[1], L);
        uint32_t cz = cell_coord(p.z, b.lo[2], b.hi[2], L);
        keys[i] = morton3(cx, cy, cz);
        seq[i] = i;
    }
}

// Gather of every attribute by the sort permutation (copy_scattered_read.comp).
// With srec non-null it also writes each particle's search record (position xyz,
// fixed-point search radius R = range_fixed(kw, scale) in w, -1 for a NaN or
// negative width) and reduces the radii's range into the status block, so that the
// row build knows before it starts whether every radius is equal.
__global__ void k_reorder(FluidBufs src, FluidBufs dst, const uint32_t *perm, uint32_t *inv_perm,
                          const uint32_t *d_len, int4 *srec, float scale, Status *st) {
    grid_dependency_wait();
    grid_dependency_trigger();
    uint32_t n = d_len[kLenParticles];
    long long rmin = 0x7fffffffffffffffll, rmax = -1;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        uint32_t o = perm[k];
        int4 p = src.pos[o];
        p.w = __float_as_int(1.0f / src.inv_mass[o]);  // the solver's per-particle mass (position.w is reserved)
        dst.pos[k] = p;
        dst.vel[k] = src.vel[o];
        dst.inv_mass[k] = src.inv_mass[o];
        dst.radius[k] = src.radius[o];
        dst.pos_backup[k] = src.pos_backup[o];
        dst.transferring[k] = src.transferring[o];
        dst.target_radius[k] = src.target_radius[o];
        dst.kernel_width[k] = src.kernel_width[o];
        dst.boundariness[k] = src.boundariness[o];
        dst.lambda_prev[k] = src.lambda_prev[o];
        dst.boundary_distance[k] = src.boundary_distance[o];
        inv_perm[o] = k;
        if (srec) {
            const long long R = range_fixed(src.kernel_width[o], scale);
            srec[k] = make_int4(p.x, p.y, p.z, (int)R);
            if (R >= 0) {
                rmin = R < rmin ? R : rmin;
                rmax = R > rmax ? R : rmax;
            }
        }
    }
    if (!srec) return;  // uniform over the grid
    for (int off = 16; off > 0; off >>= 1) {
        const long long a2 = __shfl_down_sync(0xffffffffu, rmin, off);
        const long long c2 = __shfl_down_sync(0xffffffffu, rmax, off);
        rmin = a2 < rmin ? a2 : rmin;
        rmax = c2 > rmax ? c2 : rmax;
    }
    // a bound that already holds is left alone: every write of these two words passes
    // between the SMs, a read does not
    if ((threadIdx.x & 31) == 0 && rmax >= 0) {
        if ((unsigned long long)rmin < *(volatile unsigned long long *)&st->range_min)
            atomicMin(&st->range_min, (unsigned long long)rmin);
        if ((unsigned long long)rmax > *(volatile unsigned long long *)&st->range_max)
            atomicMax(&st->range_max, (unsigned long long)rmax);
    }
}

// find_value_ranges.comp:15-31 (cell arrays zeroed beforehand).
// The transfer list follows the reorder here as well.
__global__ void k_cell_ranges(const uint32_t *skeys, const uint32_t *d_len, uint32_t *start, uint32_t *end,
                              TransferBufs tr, const uint32_t *inv_perm, Status *st) {
    grid_dependency_wait();
    grid_dependency_trigger();
    uint32_t n = d_len[kLenParticles];
    remap_transfers(tr, inv_perm, d_len, st);
    for (uint32_t id = blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
        uint32_t cur = skeys[id];
        uint32_t prev = id == 0 ? cur : skeys[id - 1];
        if (id == 0 || cur != prev) start[cur] = id;
        if (id != 0 && cur != prev) end[prev] = id;
        if (id == n - 1) end[cur] = id + 1u;
    }
}

struct BuildArgs {
    const int4 *pos;
    int4 *pos_box;  // when non-null: receives box_collision(pos) (the first Jacobi iteration's box pass)
    const float *radius;
    const float4 *bmin, *bmax, *rot;
    uint32_t nboxes;
    const uint32_t *d_len;
    Bounds b;
    uint32_t L;
    int fast_ok;  // the grid spans less than 2^31 units on every axis, within the range of 32 bits
    const uint32_t *cstart, *cend;
    uint32_t stride, maxn;
    uint32_t *count, *idx;
    unsigned long long *total;
    Status *st;
    const int4 *srec;         // per particle: position xyz and fixed-point search radius R (w)
    uint32_t *ucount, *uidx;  // correction rows (the reverse-row arrays), when the radii differ
    uint32_t *one_sided;      // per particle: one-sided pairs of its row (radii that differ)
    int corrections;          // 0: no correction rows (the caller transposes pruned rows next)
};

// Appends an entry to a correction row (the reverse-row arrays; their counts were
// zeroed by the walk, and any row may append, so the slot is an atomic).
__device__ __forceinline__ void push_correction(const BuildArgs &a, uint32_t row, uint32_t entry) {
    const uint32_t slot = atomicAdd(&a.ucount[row], 1u);
    if (slot < a.maxn) {
        a.uidx[(size_t)slot * a.stride + row] = entry;
    } else {
        set_flag(a.st, APBF_FLAG_NEIGHBOR_OVERFLOW);
        atomicMax(&a.st->required_neighbors, slot + 1u);
    }
}

// The one-sided pairs of the rows just built (radii that differ; particles whose
// walk counted some): found again on the particle's row, i's correction row
// subtracts j, j's adds i.  A kernel of its own, so that the walk holds no atomics.
__global__ void k_corrections(BuildArgs a) {
    grid_dependency_wait();
    grid_dependency_trigger();
    if (!a.corrections || a.st->range_min == a.st->range_max) return;  // none wanted, or nothing one-sided
    const uint32_t n = a.d_len[kLenParticles];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (!a.one_sided[i]) continue;
        const int4 p = a.srec[i];
        const uint32_t m = a.count[i];
        for (uint32_t k = 0; k < m; ++k) {
            const uint32_t j = a.idx[(size_t)k * a.stride + i];
            const int4 q = a.srec[j];
            const unsigned long long Rj = (unsigned long long)(uint32_t)max(q.w, 0);
            if (q.w >= 0 && dist2_within<false>(p, q, (uint32_t)Rj) <= Rj * Rj) continue;
            push_correction(a, i, j | kNoDelta);
            push_correction(a, j, i);
        }
    }
}

// The rows (neighborhood_green.comp:49-87 with the canonical predicate, C2): G threads
// walk the cells around one particle and append every j != i with |x_j - x_i| <= R_i, cells
// in z, y, x order and their particles in list order.
//
// A thread per particle (as this kernel once was) is a chain of dependent loads, 120 us
// however few the particles (now 12 us at 2 197, 39 at 32 768), and idles at 12 of 32 lanes
// where their cells differ in length (the drop of 250 000: 260 against 176 us, the waterfall's
// million: 795 against 576; bound by instruction issue).  Here a group's threads load the
// ranges of G pairs of cells at once and then test the joined ranges together (RowWalk).
//
// Correction rows (uni, when the search radii differ): the position update of
// particle i sums over the particles k whose rows hold i (|x_i - x_k| <= R_k),
// and its deferred boundariness filter tests i's own row.  It sums over i's own
// row and then over i's correction row: entries j of i's row whose radius does not
// reach i (flagged kNoDelta, their terms subtracted), and particles k whose rows
// hold i although i's radius does not reach them (added).  Both kinds are one-sided
// pairs, counted here (one_sided) and appended by k_corrections.

// c / d of small numbers: d at most 512 and c below 2^22 by one product, exactly.
struct SmallDiv {
    uint32_t d, inv;
    __device__ __forceinline__ explicit SmallDiv(uint32_t d_) : d(d_), inv(0xffffffffu / d_ + 1u) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t c, bool big) const {
        if (big) return c / d;
        return d == 1u ? c : __umulhi(c, inv);
    }
};

// The cells of a particle's box axis by axis: pairs along x, then cells along y and z.
struct CellBox {
    uint32_t x0, y0, z0, nx, ny;
    bool inside;  // the box touches no edge cell of the grid
};
// Cell e of that list: how far the particle is from it along its axis (0 when the box is not
// inside the grid) and its share of the key.
__device__ __forceinline__ uint2 axis_cell(const Bounds &b, uint32_t L, const CellBox &box, int4 p, uint32_t e) {
    const uint32_t d = e < box.nx ? 0u : e < box.nx + box.ny ? 1u : 2u;
    const uint32_t c = d == 0u ? 2u * ((box.x0 >> 1) + e) : d == 1u ? box.y0 + (e - box.nx) : box.z0 + (e - box.nx - box.ny);
    uint32_t gap = 0u;
    if (box.inside) {
        const int x = d == 0u ? p.x : d == 1u ? p.y : p.z;
        const long long lo64 = d == 0u ? b.lo[0] : d == 1u ? b.lo[1] : b.lo[2];
        const uint32_t span = (uint32_t)((d == 0u ? b.hi[0] : d == 1u ? b.hi[1] : b.hi[2]) - lo64);
        const int lo = (int)lo64;
        const int first = lo + (int)(((unsigned long long)c * span) >> L),
                  behind = lo + (int)(((unsigned long long)(c + (d == 0u ? 2u : 1u)) * span) >> L);
        gap = (uint32_t)max(max(first - x, x - behind), 0);
    }
    return make_uint2(gap, spread3(c) << d);
}

// The cells are taken in pairs along x: cells 2k and 2k + 1 have neighbouring keys, so their
// particles are one run, in the order the cells would give.  Pairs that lie beyond the
// radius (a lower bound of the distance from the pair's box) bring nothing; a quarter of
// the candidates are in such cells.
// A pair's distance and key come from a table of the box's cells per axis: worked out anew for
// every pair they were half of a sparse list's instructions (a million particles with 14
// neighbours each 825 us, 640 with the table; with 6 each 507 and 428; the thread per particle
// took 745 and 364).  The table holds boxes of up to 17 cells an axis; larger ones do without.
constexpr uint32_t kAxisCells = 48;  // cells along x (pairs), y and z together
template <int G>
__global__ void __launch_bounds__(kBuildThreads, 6) k_build_rows(BuildArgs a) {
    constexpr uint32_t P = RowWalk<G>::kParticles;
    __shared__ uint32_t s_row[kRowStage * RowWalk<G>::kPad];
    __shared__ uint32_t s_cnt[P];
    __shared__ uint2 s_axis[P * kAxisCells];
    grid_dependency_wait();
    grid_dependency_trigger();
    const uint32_t n = a.d_len[kLenParticles];
    const uint32_t last = (1u << a.L) - 1u;
    const bool uni = a.corrections && a.st->range_min != a.st->range_max;  // the radii differ: correction rows
    if (blockIdx.x == 0 && threadIdx.x == 0) a.st->union_rows = uni ? 1u : 0u;
    RowWalk<G> w(a.srec, a.idx, a.stride, a.maxn, s_row, uni);
    const uint32_t gl = w.gl;
    unsigned long long local = 0;
    for (uint32_t base = blockIdx.x * P; base < n; base += gridDim.x * P) {
        const uint32_t i = base + w.slot;
        const bool valid = i < n;
        const int4 p = valid ? a.srec[i] : make_int4(0, 0, 0, -1);
        const long long R = p.w;
        // the six faces of the cell box, a thread each
        uint32_t face = 0;
        if (R >= 0 && gl < 6u) {
            const uint32_t d = gl >> 1;
            const long long x = d == 0u ? p.x : d == 1u ? p.y : p.z;
            const long long lo = d == 0u ? a.b.lo[0] : d == 1u ? a.b.lo[1] : a.b.lo[2];
            const long long hi = d == 0u ? a.b.hi[0] : d == 1u ? a.b.hi[1] : a.b.hi[2];
            face = cell_coord((gl & 1u) ? x + R : x - R, lo, hi, a.L);
        }
        const uint32_t x0 = __shfl_sync(0xffffffffu, face, 0, G), x1 = __shfl_sync(0xffffffffu, face, 1, G),
                       y0 = __shfl_sync(0xffffffffu, face, 2, G), y1 = __shfl_sync(0xffffffffu, face, 3, G),
                       z0 = __shfl_sync(0xffffffffu, face, 4, G), z1 = __shfl_sync(0xffffffffu, face, 5, G);
        if (valid && R < 0 && gl == 0u) set_flag(a.st, APBF_FLAG_NONFINITE);  // NaN or negative width: no neighbours
        const uint32_t nx = (x1 >> 1) - (x0 >> 1) + 1u, ny = y1 - y0 + 1u, nz = z1 - z0 + 1u;
        const uint32_t npair = R < 0 ? 0u : nx * ny * nz;
        // A box that touches no edge cell of the grid only meets particles inside the grid
        // (edge cells also hold the clamped outsiders): 32-bit differences.
        const bool fast = a.fast_ok && x0 > 0 && y0 > 0 && z0 > 0 && x1 < last && y1 < last && z1 < last;
        const bool all_fast = __all_sync(0xffffffffu, fast || npair == 0u);
        w.start(i, p, (uint32_t)max(p.w, 0));
        const bool big = npair >= (1u << 22);
        const SmallDiv by_x(nx), by_y(ny);
        const CellBox box = {x0, y0, z0, nx, ny, fast};
        uint2 *axis = s_axis + w.slot * kAxisCells;
        const uint32_t ncells = npair == 0u ? 0u : nx + ny + nz;
        const uint32_t most = __reduce_max_sync(0xffffffffu, npair);  // the warp's groups go on together
        // gap of a coordinate to cells [c, e) of an axis (inside the grid), where the table is too short
        const auto gap = [&](int x, int d, uint32_t c, uint32_t e) {
            const uint32_t span = (uint32_t)(a.b.hi[d] - a.b.lo[d]);
            const int lo = (int)a.b.lo[d];
            const int first = lo + (int)(((unsigned long long)c * span) >> a.L),
                      behind = lo + (int)(((unsigned long long)e * span) >> a.L);
            return (uint32_t)max(max(first - x, x - behind), 0);
        };
        const auto walk = [&](auto tabled) {
            const auto range = [&](uint32_t c, uint32_t &s, uint32_t &len) {  // of the c-th pair of the box
                s = len = 0u;
                if (c >= npair) return;
                const uint32_t t = by_x(c, big), u = by_y(t, big), ix = c - t * nx, iy = t - u * ny;
                const uint32_t cx = 2u * ((x0 >> 1) + ix);
                uint32_t gx = 0u, gy = 0u, gz = 0u, key;
                if (decltype(tabled)::value) {
                    const uint2 ex = axis[ix], ey = axis[nx + iy], ez = axis[nx + ny + u];
                    gx = ex.x;
                    gy = ey.x;
                    gz = ez.x;
                    key = ex.y | ey.y | ez.y;
                } else {
                    const uint32_t cy = y0 + iy, cz = z0 + u;
                    if (all_fast) {
                        gx = gap(p.x, 0, cx, cx + 2u);
                        gy = gap(p.y, 1, cy, cy + 1u);
                        gz = gap(p.z, 2, cz, cz + 1u);
                    }
                    key = morton3(cx, cy, cz);
                }
                if ((unsigned long long)gx * gx + (unsigned long long)gy * gy + (unsigned long long)gz * gz > w.R2) return;
                const uint2 st = *reinterpret_cast<const uint2 *>(a.cstart + key), en = *reinterpret_cast<const uint2 *>(a.cend + key);
                const uint32_t n0 = cx >= x0 ? en.x - st.x : 0u, n1 = cx + 1u <= x1 ? en.y - st.y : 0u;
                s = n0 ? st.x : st.y;
                len = n0 + n1;
            };
            uint32_t s, len;
            range(gl, s, len);
            for (uint32_t c0 = 0; c0 < most; c0 += G) {
                uint32_t ns, nlen;
                range(c0 + G + gl, ns, nlen);  // in flight while this round's candidates are tested
                if (all_fast) w.template take<true>(s, len);
                else w.template take<false>(s, len);
                s = ns;
                len = nlen;
            }
        };
        if (__all_sync(0xffffffffu, ncells <= kAxisCells)) {
            for (uint32_t e = gl; e < ncells; e += G) axis[e] = axis_cell(a.b, a.L, box, p, e);
            __syncwarp();
            walk(std::true_type());
        } else {
            walk(std::false_type());
        }
        if (uni) {
            const uint32_t one_sided = group_total<G>(w.one_sided);
            if (valid && gl == 0u) a.one_sided[i] = one_sided;  // k_corrections appends them
        }
        if (gl == 0u) {
            const uint32_t kept = min(w.count, a.maxn);
            s_cnt[w.slot] = kept;
            if (valid) {
                a.ucount[i] = 0u;  // no correction rows yet
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
        if (a.pos_box && threadIdx.x < P && base + threadIdx.x < n) {
            const uint32_t k = base + threadIdx.x;
            a.pos_box[k] = box_push_call(a.pos[k], a.radius[k], k, a.bmin, a.bmax, a.rot, a.nboxes);
        }
        __syncthreads();  // the rows are the next particles'
    }
    add_pairs(a.total, local);
}

__global__ void k_reverse_rows(const uint32_t *d_len, uint32_t stride, uint32_t maxn, const uint32_t *__restrict__ count,
                               const uint32_t *__restrict__ idx, uint32_t *__restrict__ rcount,
                               uint32_t *__restrict__ ridx, Status *st) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->union_rows = 0u;
    if (st->range_min == st->range_max) return;  // symmetric rows: reverse = forward
    uint32_t n = d_len[kLenParticles];
    // four entries per batch: their slot atomics are in flight together (the slots'
    // order within a reverse row is arbitrary either way, and the position update's
    // integer sums do not depend on it)
    constexpr uint32_t U = 4;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = count[i];
        for (uint32_t k0 = 0; k0 < c; k0 += U) {
            uint32_t j[U], slot[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) j[u] = k0 + u < c ? idx[(size_t)(k0 + u) * stride + i] : 0u;
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) slot[u] = k0 + u < c ? atomicAdd(&rcount[j[u]], 1u) : 0u;
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                if (k0 + u >= c) break;
                if (slot[u] < maxn) {
                    ridx[(size_t)slot[u] * stride + j[u]] = i;
                } else {
                    set_flag(st, APBF_FLAG_NEIGHBOR_OVERFLOW);
                    atomicMax(&st->required_neighbors, slot[u] + 1u);
                }
            }
        }
    }
}

__global__ void k_clamp_rev(const uint32_t *d_len, uint32_t maxn, uint32_t *rcount, Status *st) {
    grid_dependency_wait();
    grid_dependency_trigger();
    if (st->range_min == st->range_max) return;
    uint32_t n = d_len[kLenParticles];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (rcount[i] > maxn) rcount[i] = maxn;
}

// Pair export (the reference's uvec2 list): row-major order of the rows.
__global__ void k_export_pairs(const uint32_t *d_len, uint32_t stride, const uint32_t *__restrict__ count,
                               const uint32_t *__restrict__ idx, const uint32_t *__restrict__ offsets, uint32_t cap,
                               uint2 *__restrict__ out) {
    uint32_t n = d_len[kLenParticles];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t c = count[i];
        uint32_t o = offsets[i] - c;  // inclusive scan -> row start
        for (uint32_t k = 0; k < c; ++k)
            if (o + k < cap) out[o + k] = make_uint2(i, idx[(size_t)k * stride + i]);
    }
}

__global__ void k_export_len(const uint32_t *d_len, const uint32_t *offsets, uint32_t *out_len) {
    uint32_t n = d_len[kLenParticles];
    *out_len = n ? offsets[n - 1] : 0u;
}

void swap_all(apbf_ctx *ctx) { ctx->fcur ^= 1; }

}  // namespace

// Gathers every particle attribute in the order ctx->perm gives (new id -> old id),
// remaps the glue list, and makes the gathered set current; the transfer list is left to
// the caller's next kernel (remap_transfers with ctx->inv_perm).
// With `search` the gather also writes the search records (srec) for range scale
// `scale` and reduces the search radii's range into the status block.
apbf_status reorder_particles(apbf_ctx *ctx, cudaStream_t s, bool search, float scale, bool behind) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    FluidBufs &cur = ctx->fl[ctx->fcur];
    FluidBufs &alt = ctx->fl[ctx->fcur ^ 1];
    APBF_BEFORE_LAUNCH(ctx, s, "k_reorder");
    APBF_CUDA(launch_behind(behind, k_reorder, grid_for(ctx, cap), kBlock, 0, s, cur, alt, ctx->perm, ctx->inv_perm,
                            ctx->d_len, search ? ctx->srec : nullptr, scale, ctx->status));
    APBF_AFTER_LAUNCH(ctx, s, "k_reorder");
    apbf_status r = glue_remap(ctx, s);
    if (r != APBF_OK) return r;
    swap_all(ctx);
    return APBF_OK;
}

apbf_status neighborhood_green(apbf_ctx *ctx, float range_scale, const float minp[3], const float maxp[3],
                               uint32_t L, cudaStream_t s, bool fuse_box, bool corrections) {
    if (L < 1 || L > ctx->cfg.max_log2res || L > 10) {
        set_error("neighborhood_green: log2res must be in [1, max_log2res of apbf_create]");
        return APBF_ERR_INVALID_ARG;
    }
    const uint32_t cap = ctx->cfg.particle_capacity;
    Bounds b = fixed_bounds(minp, maxp);
    FluidBufs &cur = ctx->fl[ctx->fcur];
    const int g = grid_for(ctx, cap);
    const size_t ncells = (size_t)1 << (3 * L);
    uint32_t *cell_start = ctx->cells, *cell_end = ctx->cells + ncells;
    // cleared ahead, so that from the sort on kernel follows kernel and each starts as the one
    // before it ends (19 683 particles stage by stage 202 -> 194 us, 2 197 143 -> 136 a frame,
    // 250 000 1357 -> 1344; not in a batch, whose waiting blocks would keep
    // other scenes' off the SMs)
    const bool behind = !ctx->in_batch;
    APBF_CUDA(cudaMemsetAsync(ctx->cells, 0, 2 * ncells * sizeof(uint32_t), s));
    APBF_BEFORE_LAUNCH(ctx, s, "k_position_keys");
    k_position_keys<<<g, kBlock, 0, s>>>(cur.pos, ctx->d_len, b, L, ctx->keys[0], ctx->vals[0], ctx->status,
                                         ctx->d_pairs);
    APBF_AFTER_LAUNCH(ctx, s, "k_position_keys");
    apbf_status r = sort_pairs_device(ctx, ctx->keys[0], ctx->vals[0], ctx->d_len + kLenParticles, cap, 3u * L,
                                      ctx->sorted_keys, ctx->perm, s, nullptr, true);
    if (r != APBF_OK) return r;
    r = reorder_particles(ctx, s, true, range_scale, behind);
    if (r != APBF_OK) return r;
    FluidBufs &f = ctx->fl[ctx->fcur];

    APBF_BEFORE_LAUNCH(ctx, s, "k_cell_ranges");
    APBF_CUDA(launch_behind(behind, k_cell_ranges, g, kBlock, 0, s, ctx->sorted_keys, ctx->d_len, cell_start, cell_end,
                            ctx->tr[ctx->tcur], ctx->inv_perm, ctx->status));
    APBF_AFTER_LAUNCH(ctx, s, "k_cell_ranges");
    APBF_BEFORE_LAUNCH(ctx, s, "k_build_rows");
    BuildArgs ba;
    ba.pos = f.pos;
    FluidBufs &spare = ctx->fl[ctx->fcur ^ 1];
    ba.pos_box = fuse_box ? spare.pos : nullptr;
    ba.radius = f.radius;
    ba.bmin = ctx->box_min;
    ba.bmax = ctx->box_max;
    ba.rot = ctx->box_rot;
    ba.nboxes = ctx->n_boxes;
    ba.d_len = ctx->d_len;
    ba.b = b;
    ba.L = L;
    ba.fast_ok = 1;
    for (int d = 0; d < 3; ++d)
        if (b.hi[d] - b.lo[d] >= (1ll << 31) || b.lo[d] < -(1ll << 31) || b.hi[d] >= (1ll << 31)) ba.fast_ok = 0;
    ba.cstart = cell_start;
    ba.cend = cell_end;
    ba.stride = ctx->row_stride;
    ba.maxn = ctx->cfg.max_neighbors;
    ba.count = ctx->nb_count;
    ba.idx = ctx->nb_idx;
    ba.total = ctx->d_pairs;
    ba.st = ctx->status;
    ba.srec = ctx->srec;
    ba.ucount = ctx->rev_count;
    ba.uidx = ctx->rev_idx;
    ba.one_sided = ctx->flag_scan;  // scratch: not in use during the search
    ba.corrections = corrections ? 1 : 0;
    // threads per particle: as many as it takes to fill the chip, since a smaller group
    // shares less of its steps' fixed cost.  8 / 16 / 32 threads (cells not yet in pairs):
    // 28 / 21 / 17 us at 2 197 particles, 60 / 55 / 60 at 32 768, 206 / 222 / 290 at 250 000,
    // 663 / 794 / 1087 at a million
    if (cap <= 12288u)
        APBF_CUDA(launch_behind(behind, k_build_rows<32>, grid_for(ctx, cap, kBuildThreads / 32, 64), kBuildThreads, 0, s, ba));
    else if (cap <= 98304u)
        APBF_CUDA(launch_behind(behind, k_build_rows<16>, grid_for(ctx, cap, kBuildThreads / 16, 64), kBuildThreads, 0, s, ba));
    else
        APBF_CUDA(launch_behind(behind, k_build_rows<8>, grid_for(ctx, cap, kBuildThreads / 8, 64), kBuildThreads, 0, s, ba));
    APBF_AFTER_LAUNCH(ctx, s, "k_build_rows");
    if (corrections) {
        APBF_BEFORE_LAUNCH(ctx, s, "k_corrections");
        APBF_CUDA(launch_behind(behind, k_corrections, grid_for(ctx, cap), kBlock, 0, s, ba));
        APBF_AFTER_LAUNCH(ctx, s, "k_corrections");
    }
    if (fuse_box) {  // the box-collided positions are the current ones now
        int4 *t = f.pos;
        f.pos = spare.pos;
        spare.pos = t;
    }
    if (corrections) {
        APBF_BEFORE_LAUNCH(ctx, s, "k_clamp_rev");
        APBF_CUDA(launch_behind(behind, k_clamp_rev, grid_for(ctx, cap), kBlock, 0, s, ctx->d_len,
                                ctx->cfg.max_neighbors, ctx->rev_count, ctx->status));
        APBF_AFTER_LAUNCH(ctx, s, "k_clamp_rev");
    }
    return APBF_OK;
}

// Reverse rows by transposing the forward rows (the binary-search neighbourhood and
// the rows spread_kernel_width prunes): row j lists every i whose row holds j, with
// no forward prefix, so the boundariness filter stays in the density pass
// (status union_rows = 0).
apbf_status build_reverse_rows(apbf_ctx *ctx, cudaStream_t s) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    APBF_CUDA(cudaMemsetAsync(ctx->rev_count, 0, (size_t)cap * sizeof(uint32_t), s));
    APBF_BEFORE_LAUNCH(ctx, s, "k_reverse_rows");
    k_reverse_rows<<<grid_for(ctx, cap), kBlock, 0, s>>>(ctx->d_len, ctx->row_stride, ctx->cfg.max_neighbors,
                                                         ctx->nb_count, ctx->nb_idx, ctx->rev_count, ctx->rev_idx,
                                                         ctx->status);
    APBF_AFTER_LAUNCH(ctx, s, "k_reverse_rows");
    APBF_BEFORE_LAUNCH(ctx, s, "k_clamp_rev");
    k_clamp_rev<<<grid_for(ctx, cap), kBlock, 0, s>>>(ctx->d_len, ctx->cfg.max_neighbors, ctx->rev_count, ctx->status);
    APBF_AFTER_LAUNCH(ctx, s, "k_clamp_rev");
    return APBF_OK;
}

apbf_status export_pairs(apbf_ctx *ctx, uint32_t *d_pairs, uint32_t cap_pairs, uint32_t *d_length, cudaStream_t s) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    APBF_CUDA(cudaMemcpyAsync(ctx->scan_tmp, ctx->nb_count, (size_t)cap * 4, cudaMemcpyDeviceToDevice, s));
    apbf_status r = prefix_sum_device(ctx, ctx->scan_tmp, ctx->d_len + kLenParticles, cap, s);
    if (r != APBF_OK) return r;
    k_export_pairs<<<grid_for(ctx, cap), kBlock, 0, s>>>(ctx->d_len, ctx->row_stride, ctx->nb_count, ctx->nb_idx,
                                                         ctx->scan_tmp, cap_pairs, (uint2 *)d_pairs);
    APBF_AFTER_LAUNCH(ctx, s, "k_export_pairs");
    APBF_BEFORE_LAUNCH(ctx, s, "k_export_len");
    k_export_len<<<1, 1, 0, s>>>(ctx->d_len, ctx->scan_tmp, d_length);
    APBF_AFTER_LAUNCH(ctx, s, "k_export_len");
    return APBF_OK;
}

}  // namespace apbf
