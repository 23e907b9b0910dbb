// solver.cu -- incompressibility::apply (source/incompressibility.cpp:12-45), one
// Jacobi iteration in two gather passes instead of the reference's four
// dispatches with per-pair integer atomics:
//
//  k_density_lambda (particle i, over its own row):  incompressibility_0.comp
//    (self density) + incompressibility_1.comp (density, weighted gradient and
//    squared-gradient sums, as 2^18 fixed-point integers) + incompressibility_2.comp
//    (lambda, boundariness, self shift) + the boundariness filter of
//    incompressibility_3.comp:41-46,60.  Writes lambda, the self shift, the
//    per-particle Gauss constants and the density-error partials (64-bit
//    fixed-point integers, turned into the FP64 mean by the position update).
//  k_delta (particle j, over the particles whose rows contain j):
//    incompressibility_3.comp:62-66 as a gather: x_j += sum_i int(gradW_ij * lambda_i * 2^18)
//    plus the self shift, into the other position buffer.
//
// The per-pair integer terms are computed by the same code from the same inputs
// as the scatter form, and integer addition is associative, so the gather is
// bit-identical to the atomic scatter.  Gradients are recomputed in k_delta
// rather than stored (the reference writes 16 bytes per pair).
//
// A substep's passes run over tiles of particles (k_density_tiles, k_delta_tiles: the
// same terms and sums from shared memory); the direct kernels serve the stage calls, the
// warm start's feature pass and short solves.
#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "apbf_internal.cuh"

namespace apbf {
namespace {

// Contraction-proof dot product: k_density_lambda and k_delta must evaluate
// bit-identical gradients for the same pair.
__device__ __forceinline__ float dot3x(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}

// The boundariness filter of incompressibility_3.comp:41-46,60 for the Gauss
// kernel, whose gradient points along -d: the pair (i, j) at offset d = x_j - x_i
// clears a non-zero boundariness of i when -normalize(gradW) . ed > 0.6 with
// ed = -normalize(gradient sum of i).  Explicit rounding: the density pass and the
// position pass (which takes the test over when rows are symmetric) must agree.
__device__ __forceinline__ bool filter_dir(int32_t gx, int32_t gy, int32_t gz, float3 &ed) {
    const float3 gi = make_float3((float)gx, (float)gy, (float)gz);
    const float gl = __fsqrt_rn(dot3x(gi, gi));
    if (!(gl > 0.0f)) return false;
    ed = make_float3(-__fdiv_rn(gi.x, gl), -__fdiv_rn(gi.y, gl), -__fdiv_rn(gi.z, gl));
    return true;
}
__device__ __forceinline__ bool gauss_filter_hit(float3 ed, float3 d) {
    const float r2 = dot3x(d, d);
    if (r2 < 1.0e-8f) return false;  // zero gradient: normalize() gives NaN, no filter
    return -dot3x(ed, d) > __fmul_rn(0.6f, __fsqrt_rn(r2));
}

struct PassA {
    const int4 *pos;
    const float *inv_mass;
    const float *radius;
    const float *kw;
    float *bness;
    const uint32_t *count;
    const uint32_t *idx;
    uint32_t stride;
    float *lambda;  // non-null (debug): the pass's lambda
    int4 *shift;
    float4 *rec;  // per particle: lambda, Gauss ivd, Gauss norm, kernel width (read by k_delta)
    int4 *pk;     // per particle: position xyz and the applied lambda (read by k_delta when widths are uniform)
    float2 *kc;   // per particle: Gauss constants of its width, ivd 2^-36 and norm (read by k_delta when widths differ)
    uint32_t *dbg_dens;
    int4 *dbg_grad;
    uint32_t *dbg_sq;
    PassSync *sync;       // the pass's error sums (2^-24 fixed point) and width uniformity, for the position update
    const uint32_t *d_len;
    Status *st;
    double *red_out;     // [2], [3]: mean compression / absolute error of this pass
    float *features;     // non-null: the 8 features of this pass (first pass of a substep)
    float4 *selfdir;     // non-null with features: self-shift direction and inverse mass
    const float4 *vel;   // velocities, for the divergence feature
    const float *lam_prev;  // lambda_prev: the previous substep's sum at pass 0, this substep's after
    int projected;          // 1: pull-back allowed (passes after the first of a warm-started substep)
    int loop_offset;        // >= 0: solve loop pass number = st->pass_start + loop_offset
    uint32_t max_passes;    // loop passes from this number on are skipped
    int4 *filt;             // non-null: Gauss filter deferred to the position pass when rows are symmetric
    float target;        // > 0: set st->converged when the error is at most this
    uint32_t target_m;   //   = target_m 2^-(target_s + 24) (split_target)
    int target_s;
    int early_exit;      // skip the pass when st->converged is set
    float rmin3;  // pow(2 * smallestTargetRadius, 3)
    int hk, gk, method, update_b;
    float one;  // 1, as a value that is not known before the launch (see F2)
    float b_speed, b_sgl_factor, b_up_factor;
};

// Gauss constants in the units of the unscaled fixed-point offset D (2^18 per
// reference unit): the exponent scale ivd 2^-36 (r^2 = |D|^2 2^-36), the height
// norm, and the gradient factor 2 ln2 ivd 2^-18 (kernels.glsl:112-123 with r = D 2^-18).
struct GaussPair {
    float ivd36, norm, k2;
};
__device__ __forceinline__ GaussPair gauss_pair(float ivd36, float norm) {
    // k2 = round(ivd ln2) 2^-17: the factor 2 of the gradient and the 2^-18 of r = D 2^-18
    return {ivd36, norm, ivd36 * (0.693147180559945309f * 0x1p19f)};
}
__device__ __forceinline__ GaussPair gauss_pair(KConst c) { return gauss_pair(c.ivd * 0x1p-36f, c.norm); }
__device__ __forceinline__ float3 udiff(int4 from, int4 to) {
    return make_float3((float)wadd(to.x, -from.x), (float)wadd(to.y, -from.y), (float)wadd(to.z, -from.z));
}

// The Gauss height and gradient of the offset D = to - from in fixed-point units.
// Every product is the FP32 rounding of the reference-unit product (fdiff, r2,
// kernel_gradient's -2 ivd W r) scaled by a power of two, which is exact in the
// normal range: the terms equal the reference-unit evaluation bit for bit, except
// for gradients far below one fixed-point unit of any sum (subnormal intermediates).
__device__ __forceinline__ void gauss_terms_r2(float3 D, float r2, const GaussPair &k, float &W, float3 &g) {
    W = exp2f(r2 * k.ivd36) * k.norm;
    if (r2 < 1.0e-8f * 0x1p36f) {  // dist < 0.0001 reference units
        g = make_float3(0.f, 0.f, 0.f);
        return;
    }
    const float s = W * k.k2;
    g = make_float3(s * D.x, s * D.y, s * D.z);
}
__device__ __forceinline__ void gauss_terms(float3 D, const GaussPair &k, float &W, float3 &g) {
    gauss_terms_r2(D, dot3x(D, D), k, W, g);
}

// gauss_filter_hit for the offset x_j - x_i = -D, D in fixed-point units and
// r2 = |D|^2.  Every quantity is the reference-unit one times a power of two, and
// none is subnormal (|D| components are 0 or >= 1, those of ed 0 or >= 2^-32), so
// the decision is gauss_filter_hit's bit for bit.
__device__ __forceinline__ bool gauss_filter_hit_fixed(float3 ed, float3 D, float r2) {
    if (r2 < 1.0e-8f * 0x1p36f) return false;
    return dot3x(ed, D) > __fmul_rn(0.6f, __fsqrt_rn(r2));
}

template <bool GAUSS>
__device__ __forceinline__ void pair_terms(int hk, int gk, float3 d, float kw, KConst c, float &W, float3 &g) {
    float r2 = dot3x(d, d);
    if (GAUSS) {
        W = gauss_height(r2, c);
        g = kernel_gradient(1, d, r2, kw, c, W);
    } else {
        W = kernel_height(hk, r2, kw, c);
        float Wg = gk == 1 ? (hk == 1 ? W : gauss_height(r2, c)) : 0.0f;
        g = kernel_gradient(gk, d, r2, kw, c, Wg);
    }
}

// Fixed-order (deterministic) sum of per-block partial pairs with one block of
// blockDim.x (a power of two, at most 256) threads: thread t sums partials t,
// t + blockDim.x, ... in order, then a fixed tree.
__device__ __forceinline__ void block_sum2(const double *partials, int blocks, double &t1, double &t2) {
    __shared__ double s1[256], s2[256];
    double a = 0.0, b = 0.0;
    for (int k = threadIdx.x; k < blocks; k += blockDim.x) {
        a += ((volatile const double *)partials)[2 * k];
        b += ((volatile const double *)partials)[2 * k + 1];
    }
    s1[threadIdx.x] = a;
    s2[threadIdx.x] = b;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) {
            s1[threadIdx.x] += s1[threadIdx.x + off];
            s2[threadIdx.x] += s2[threadIdx.x + off];
        }
        __syncthreads();
    }
    t1 = s1[0];
    t2 = s2[0];
}

// Mean density error terms: per particle in 2^-24 fixed point (the FP32 ratio
// times 2^24 is exact; ratios of 128 and more saturate), summed as 64-bit
// integers.  Integer sums are order-free, so the mean is deterministic without
// FP64 arithmetic per particle (GB300's FP64 pipe is a small fraction of its FP32
// rate).  NaN counts as saturated, so a NaN state never converges.
constexpr float kErrScale = 16777216.0f;
__device__ __forceinline__ long long err_fix(float x) {
    return x != x ? 0x7fffffffll : (long long)__float2int_rn(__fmul_rn(x, kErrScale));
}

constexpr int kUnroll = 4;

// L threads per particle ("lanes"): lane s of a particle's group takes row
// entries s, s + L, ...; the group's integer sums are then combined by shuffles.
// Wrapping integer sums are order-free, so every L gives the same density,
// gradient and squared-gradient sums bit for bit.
template <int L, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}
template <int L>
__device__ __forceinline__ float group_min(float v) {
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}
template <int L>
__device__ __forceinline__ int32_t group_wsum(int32_t v) {
#pragma unroll
    for (int off = L / 2; off > 0; off >>= 1) v = wadd(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

// XTRA: the warm-start features or the centre-of-mass boundariness sums
// (method 1) are gathered too; the common pass is compiled without them.
// Per-thread partial results of a density pass: the two error sums (2^-24 fixed
// point) and whether a kernel width's bits differed from kw0's.
struct PassSums {
    long long e1 = 0, e2 = 0;
    uint32_t kw0 = 0u;
    bool kw_diff = false;
};

// What a density pass has summed over one particle's row.
struct RowSums {
    uint32_t dens = 0u, sq = 0u;
    int32_t gx = 0, gy = 0, gz = 0;
    int32_t cx = 0, cy = 0, cz = 0, cw = 0;  // method 1: the centre-of-mass sums
    float div = 0.0f;    // sum_j m_j (v_j - v_i) . gradW_ij  (velocity divergence x density)
    float nprev = 0.0f;  // sum_j lambda_prev_j (the neighbours' previous-substep lambda sums)
};

// The rest of a particle's density pass once its row is summed (one thread):
// incompressibility_2.  Returns whether the boundariness filter is left to the caller
// (Gauss kernel, not deferred): a neighbour within the cone around ed clears bness[i].
template <bool GAUSS, bool XTRA>
__device__ __forceinline__ bool density_finish(const PassA &a, const int4 *pos, uint32_t i, const int4 &p, float kw,
                                               const KConst &c, const GaussPair &gp, uint32_t cnt, const RowSums &rs,
                                               float im, float radius, float b, float pushed, bool feat, bool defer,
                                               bool write_rec, PassSums &ps, float3 &ed) {
    bool ask = false;
    uint32_t dens = rs.dens;
    const uint32_t sq = rs.sq;
    const int32_t gx = rs.gx, gy = rs.gy, gz = rs.gz, cx = rs.cx, cy = rs.cy, cz = rs.cz, cw = rs.cw;
    const float div = rs.div, nprev = rs.nprev;
    const float W0 = GAUSS ? c.norm : kernel_height(a.hk, 0.0f, kw, c);
    dens += f2u(W0 / im * APBF_FIX);  // incompressibility_0.comp:32-45 (the self term)
    // incompressibility_2.comp:77-109
    const float r2x = 2.0f * radius;
    const float ird = (r2x * r2x * r2x) * im;
    const float density = (float)dens * APBF_INV_FIX;
    const float3 wgs = make_float3((float)gx * APBF_INV_FIX, (float)gy * APBF_INV_FIX, (float)gz * APBF_INV_FIX);
    float sqs = (float)sq * APBF_INV_FIX;
    const float wgsq = dot3x(wgs, wgs);
    const float sgl = sqrtf(wgsq) * ird;
    sqs += wgsq * im;
    const float under = 1.0f - density * ird;
    if (a.update_b) {
        float bn;
        if (XTRA && a.method == 1) {
            float tm = (float)cw * APBF_INV_FIX + 1.0f / im;
            float3 cv = make_float3((float)cx, (float)cy, (float)cz);
            bn = sqrtf(dot3x(cv, cv)) / (APBF_FIX * tm) * a.b_sgl_factor;
        } else {
            bn = sgl * kw * a.b_sgl_factor + fmaxf(0.0f, under) * a.b_up_factor;
        }
        bn = bn >= 1.0f ? 1.0f : 0.0f;
        float step = bn - b;
        b = b + fminf(a.b_speed, fmaxf(-a.b_speed, step));
        b = fminf(1.0f, b);
    }
    float lam = under / (ird * ird * (sqs + 0.01f));
    lam /= a.rmin3 / ird * im;
    if (a.lambda) a.lambda[i] = lam;
    // The lambda this pass applies: the reference applies only pushes (lambda < 0,
    // incompressibility_2.comp:106, incompressibility_3.comp:63).  Projected mode
    // (warm-started solve) also applies a pull-back lambda > 0 where earlier passes
    // of this substep pushed, up to their sum, so that an over-push is undone; the
    // density that pull-back would restore counts as error.
    float applied = lam < 0.0f ? lam : 0.0f;
    float pull = 0.0f;
    if (a.projected && lam > 0.0f) {
        applied = fminf(lam, -pushed);  // the sum applied so far (<= 0)
        if (applied > 0.0f) pull = under * (applied / lam);
        else applied = 0.0f;
    }
    if (write_rec) a.rec[i] = make_float4(applied, c.ivd, c.norm, kw);
    else if (GAUSS) a.kc[i] = make_float2(gp.ivd36, gp.norm);
    a.pk[i] = make_int4(p.x, p.y, p.z, __float_as_int(applied));
    ps.kw_diff = ps.kw_diff || __float_as_uint(kw) != ps.kw0;
    if (feat) {
        float *fo = a.features + (size_t)i * 8;
        fo[0] = (float)cnt;
        fo[1] = density * ird - 1.0f;
        fo[2] = kw / radius;
        fo[3] = lam;
        fo[4] = density > 0.0f ? div / density : 0.0f;
        fo[5] = a.lam_prev[i];
        fo[6] = cnt ? nprev / (float)cnt : 0.0f;
        fo[7] = 0.0f;
        a.selfdir[i] = make_float4(-wgs.x * ird, -wgs.y * ird, -wgs.z * ird, im);
    }
    int4 sh = make_int4(0, 0, 0, 0);
    if (applied != 0.0f) {
        const float sc = applied * im * APBF_FIX;
        sh.x = f2i(-wgs.x * ird * sc);
        sh.y = f2i(-wgs.y * ird * sc);
        sh.z = f2i(-wgs.z * ird * sc);
    } else if (!(lam >= 0.0f)) {
        set_flag(a.st, APBF_FLAG_NONFINITE);  // NaN lambda: no shift (int(NaN) = 0)
    }
    // incompressibility_3.comp:41-46,60: filter (only changes a non-zero boundariness);
    // deferred, it is recorded for particles with boundariness, flagged in shift.w
    if (defer) {
        if (b > 0.0f) {
            a.filt[i] = make_int4(gx, gy, gz, 1);
            sh.w = 1;
        }
    } else if (a.method == 2 && b > 0.0f) {
        if (GAUSS) {
            ask = filter_dir(gx, gy, gz, ed);
        } else if (!GAUSS && filter_dir(gx, gy, gz, ed)) {
            for (uint32_t k = 0; k < cnt; ++k) {
                const uint32_t j = a.idx[(size_t)k * a.stride + i];
                const float3 d = fdiff(p, pos[j]);
                {
                    float W;
                    float3 g;
                    pair_terms<GAUSS>(a.hk, a.gk, d, kw, c, W, g);
                    float l = sqrtf(dot3x(g, g));
                    if (!(l > 0.0f)) continue;
                    float dd = ed.x * (g.x / l) + ed.y * (g.y / l) + ed.z * (g.z / l);
                    if (dd > 0.6f) {
                        b = 0.0f;
                        break;
                    }
                }
            }
        }
    }
    a.shift[i] = sh;
    a.bness[i] = b;
    const float ratio = __fmaf_rn(density, ird, -1.0f);  // one rounding of the exact product - 1
    ps.e1 += err_fix(ratio > 0.0f ? ratio : pull);
    ps.e2 += err_fix(fabsf(ratio));
    if (a.dbg_dens) {
        a.dbg_dens[i] = dens;
        a.dbg_grad[i] = make_int4(gx, gy, gz, 0);
        a.dbg_sq[i] = sq;
    }
    return ask;
}

// One particle (row i_raw, lane sub of its group of L) of a density pass:
// incompressibility_0..2 and the boundariness filter of incompressibility_3.
// Every lane of the group must call it (group shuffles).
template <bool GAUSS, int L, bool XTRA>
__device__ __forceinline__ void density_one(const PassA &a, const int4 *pos, uint32_t i_raw, uint32_t n,
                                            uint32_t sub, bool defer, bool write_rec, PassSums &ps) {
    {
        const bool valid = i_raw < n;
        const uint32_t i = valid ? i_raw : 0u;
        const int4 p = pos[i];
        const float kw = a.kw[i];
        const KConst c = gauss_consts(kw);
        const GaussPair gp = gauss_pair(c);
        uint32_t dens = 0u;
        int32_t gx = 0, gy = 0, gz = 0;
        uint32_t sq = 0;
        int32_t cx = 0, cy = 0, cz = 0, cw = 0;
        const uint32_t cnt = valid ? a.count[i] : 0u;
        // loaded with the particle's other data, so that they are not one more round
        // trip after the neighbour loop
        const float im = a.inv_mass[i], radius = a.radius[i];
        const float b = a.bness[i];
        const uint32_t *row = a.idx + i;
        const bool feat = XTRA && a.features != nullptr;
        const float4 vi = feat ? a.vel[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        float div = 0.0f;  // sum_j m_j (v_j - v_i) . gradW_ij  (velocity divergence x density)
        float nprev = 0.0f;  // sum_j lambda_prev_j (the neighbours' previous-substep lambda sums)
        // Batches of kUnroll pairs per lane, software-pipelined: the neighbour gathers
        // of a batch go out with the row entries of the next, then the arithmetic, so
        // a batch costs one memory latency instead of two.
        uint32_t jj[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint32_t k = sub + u * L;
            jj[u] = k < cnt ? row[(size_t)k * a.stride] : i;
        }
        for (uint32_t k0 = sub; k0 < cnt; k0 += L * kUnroll) {
            int4 qq[kUnroll];
            uint32_t jn[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) qq[u] = pos[jj[u]];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const uint32_t k = k0 + (L * kUnroll) + u * L;
                jn[u] = k < cnt ? row[(size_t)k * a.stride] : i;
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                if (k0 + u * L >= cnt) break;
                const int4 q = qq[u];
                // the neighbour's mass rides in position.w (x / invMassN = x * mass)
                const float mjf = __int_as_float(q.w) * APBF_FIX;  // neighbour mass x 2^18
                float W;
                float3 g;
                if (GAUSS)
                    gauss_terms(udiff(p, q), gp, W, g);
                else
                    pair_terms<false>(a.hk, a.gk, fdiff(p, q), kw, c, W, g);
                dens += f2u(W * mjf);
                gx = wadd(gx, f2i(g.x * mjf));
                gy = wadd(gy, f2i(g.y * mjf));
                gz = wadd(gz, f2i(g.z * mjf));
                sq += f2u(dot3x(g, g) * mjf);
                if (feat) {
                    const float4 vj = a.vel[jj[u]];
                    div += __int_as_float(q.w) * ((vj.x - vi.x) * g.x + (vj.y - vi.y) * g.y + (vj.z - vi.z) * g.z);
                    nprev += a.lam_prev[jj[u]];
                }
                if (XTRA && a.method == 1) {  // incompressibility_1.comp:62-68
                    const float den = kw * APBF_FIX / mjf;
                    cx = wadd(cx, f2i((float)wadd(q.x, -p.x) / den));
                    cy = wadd(cy, f2i((float)wadd(q.y, -p.y) / den));
                    cz = wadd(cz, f2i((float)wadd(q.z, -p.z) / den));
                    cw = wadd(cw, f2i(mjf));
                }
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) jj[u] = jn[u];
        }
        if (L > 1) {
            dens = group_sum<L>(dens);
            sq = group_sum<L>(sq);
            gx = group_wsum<L>(gx);
            gy = group_wsum<L>(gy);
            gz = group_wsum<L>(gz);
            if (feat) {
                div = group_sum<L>(div);
                nprev = group_sum<L>(nprev);
            }
            if (XTRA && a.method == 1) {
                cx = group_wsum<L>(cx);
                cy = group_wsum<L>(cy);
                cz = group_wsum<L>(cz);
                cw = group_wsum<L>(cw);
            }
        }
        if (!valid || sub != 0) return;
        RowSums rs;
        rs.dens = dens;
        rs.sq = sq;
        rs.gx = gx;
        rs.gy = gy;
        rs.gz = gz;
        rs.cx = cx;
        rs.cy = cy;
        rs.cz = cz;
        rs.cw = cw;
        rs.div = div;
        rs.nprev = nprev;
        float3 ed;
        if (!density_finish<GAUSS, XTRA>(a, pos, i, p, kw, c, gp, cnt, rs, im, radius, b,
                                           a.projected ? a.lam_prev[i] : 0.0f, feat, defer, write_rec, ps, ed))
            return;
        // batches of kUnroll neighbours in row order, software-pipelined as the sums above
        // (the first hit ends the test, as in the plain loop)
        uint32_t fj[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) fj[u] = (uint32_t)u < cnt ? row[(size_t)u * a.stride] : i;
        bool hit = false;
        for (uint32_t k0 = 0; k0 < cnt && !hit; k0 += kUnroll) {
            int4 fq[kUnroll];
            uint32_t fn[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) fq[u] = pos[fj[u]];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const uint32_t k = k0 + kUnroll + u;
                fn[u] = k < cnt ? row[(size_t)k * a.stride] : i;
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                if (hit || k0 + u >= cnt) break;
                hit = gauss_filter_hit(ed, fdiff(p, fq[u]));
            }
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) fj[u] = fn[u];
        }
        if (hit) a.bness[i] = 0.0f;
    }
}

// Block sums of the per-thread PassSums, valid in thread 0.
__device__ __forceinline__ PassSums block_pass_sums(PassSums ps) {
    __shared__ long long s1[8], s2[8];
    for (int off = 16; off > 0; off >>= 1) {
        ps.e1 += __shfl_down_sync(0xffffffffu, ps.e1, off);
        ps.e2 += __shfl_down_sync(0xffffffffu, ps.e2, off);
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s1[w] = ps.e1;
        s2[w] = ps.e2;
    }
    PassSums t;
    t.kw_diff = __syncthreads_or(ps.kw_diff) != 0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            t.e1 += s1[k];
            t.e2 += s2[k];
        }
    }
    __syncthreads();  // the shared arrays may be reused by the next call
    return t;
}

// Adds a block's sums to the pass's (one thread).
__device__ __forceinline__ void add_pass_sums(PassSync *sync, uint32_t slot, const PassSums &bs) {
    unsigned long long *e = sync->e[slot][blockIdx.x % kSumStripes];
    if (bs.e1) atomicAdd(&e[0], (unsigned long long)bs.e1);
    if (bs.e2) atomicAdd(&e[1], (unsigned long long)bs.e2);
    if (bs.kw_diff) atomicAdd(&e[2], 1ull);
}

// The end of a density pass, once all its sums are in (one thread): mean errors,
// pass counter and, when the error met the target, the flag for the passes that follow.
__device__ __forceinline__ void finish_pass(double *red_out, Status *st, float target, uint32_t n, long long t1,
                                            long long t2, bool met) {
    const double inv = 1.0 / (double)kErrScale;
    const double m1 = n ? (double)t1 * inv / n : 0.0, m2 = n ? (double)t2 * inv / n : 0.0;
    red_out[2] = m1;
    red_out[3] = m2;
    st->density_passes += 1u;
    if (target > 0.0f && met) {
        st->converged = 1u;  // the remaining passes of the substep are skipped
        st->converged_substeps += 1u;
    }
}

// Whether a pass of the solve loop graph lies past the limit.  The body's first kernel
// reads pass_start, which its last one advances, and leaves a copy for the kernels between
// them: so no kernel writes a word that its own blocks read.
__device__ __forceinline__ bool loop_over(const PassA &a) {
    if (a.loop_offset < 0) return false;
    const uint32_t first = a.loop_offset == 0 ? a.st->pass_start : a.st->pass_index;
    if (a.loop_offset == 0 && blockIdx.x == 0 && threadIdx.x == 0) a.st->pass_index = first;
    return first + (uint32_t)a.loop_offset >= a.max_passes;
}

template <bool GAUSS, int L, bool XTRA>
__global__ void __launch_bounds__(256, GAUSS ? 4 : 3) k_density_lambda(PassA a) {
    grid_dependency_wait();
    grid_dependency_trigger();
    const bool skip = (a.early_exit && *(volatile uint32_t *)&a.st->converged) || loop_over(a);
    // With symmetric rows or union rows the Gauss filter runs in this pass's position
    // update, which gathers over the same neighbours anyway; filter_tag tells it whether to.
    const bool defer = GAUSS && a.filt && a.method == 2 &&
                       (a.st->range_min == a.st->range_max || a.st->union_rows != 0u);
    const uint32_t slot = *(volatile uint32_t *)&a.sync->cur_density & 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->filter_tag = (!skip && defer) ? 1u : 0u;
        a.sync->cur_update = slot;
    }
    if (skip) return;  // uniform over the grid
    const uint32_t n = a.d_len[kLenParticles];
    const uint32_t sub = threadIdx.x % L;
    // the position update of the Gauss kernel gathers the packed records and widths;
    // the other kernels gather the solve records, written every pass
    const bool write_rec = !GAUSS;
    PassSums ps;
    // the block iterates as a whole (uniform trip count: the group shuffles need every lane)
    const uint32_t gpb = blockDim.x / L;
    if (blockIdx.x * gpb >= n) return;  // nothing to add
    ps.kw0 = __float_as_uint(a.kw[0]);
    for (uint32_t base = blockIdx.x * gpb; base < n; base += gridDim.x * gpb)
        density_one<GAUSS, L, XTRA>(a, a.pos, base + threadIdx.x / L, n, sub, defer, write_rec, ps);
    // The block's sums go to the position update (PassSync), which waits for this kernel
    // anyway: a last block here (fence, counter, partials read back, FP64 mean) left the
    // other SMs idle for about 5 us of every pass.
    const PassSums bs = block_pass_sums(ps);
    if (threadIdx.x == 0) {
        add_pass_sums(a.sync, slot, bs);
    }
}

struct PassB {
    const int4 *pos;
    int4 *pos_out;
    const float4 *rec;
    const int4 *pk;   // the density pass's packed records (position, applied lambda)
    const float2 *kc;  // the density pass's Gauss constants per particle
    const float *kw;
    const int4 *shift;
    const float *radius;
    const float4 *bmin, *bmax, *rot;
    uint32_t nboxes;  // > 0: box collision of the next iteration applied to the output
    const uint32_t *count;
    const uint32_t *idx;
    const uint32_t *rcount;
    const uint32_t *ridx;
    uint32_t stride;
    const uint32_t *d_len;
    Status *st;
    PassSync *sync;      // this pass's error sums
    double *red_out;     // [2], [3]: mean compression / absolute error of this pass
    float target;        // > 0: the error target, target_m 2^-(target_s + 24)
    uint32_t target_m;
    int target_s;
    int gk;
    float one;  // 1, as in PassA
    int early_exit;  // converged: copy the positions unchanged (the buffers swap regardless)
    float *lam_prev;  // prev_mode / acc_mode (0 off, 1 reset, 2 add): accumulate the lambda
    float *lam_acc;   // this pass applied (rec.x: the learned one in a learned pass)
    int prev_mode, acc_mode;
    int loop_offset;      // >= 0: solve loop pass number = st->pass_index + loop_offset
    int loop_end;         // 1: the loop body's last pass, which sets the loop's condition
    cudaGraphConditionalHandle loop_handle;
    uint32_t max_passes;  // loop passes from this number on copy through; box after all but the last
    const int4 *filt;     // the density pass's deferred Gauss filter (gradient sum, boundariness > 0)
    float *bness;
};

__device__ __forceinline__ void accumulate(float *dst, int mode, uint32_t j, float v) {
    if (mode == 1) dst[j] = v;
    else if (mode == 2) dst[j] += v;
}

// One neighbour's term of a position update: int(gradW_ij * lambda_i * 2^18) per
// axis (incompressibility_3.comp:62-66) for the neighbour's record q (position,
// and for the Gauss kernel the applied lambda in w), its Gauss constants kci (as
// the density pass computed them from its width) or solve record rr.  PACKED (every
// width equal): j's own constants cj.  The main row and the correction rows use this
// one function, so a term subtracted again cancels exactly.
// The Gauss term of the offset D = x_j - x_i (fixed-point units) with r2 = |D|^2.
__device__ __forceinline__ int3 gauss_delta(float3 D, float r2, float lam, const GaussPair &k) {
    float W;
    float3 g;
    gauss_terms_r2(D, r2, k, W, g);
    const float sc = lam * APBF_FIX;
    return make_int3(f2i(g.x * sc), f2i(g.y * sc), f2i(g.z * sc));
}

template <bool GAUSS, bool PACKED>
__device__ __forceinline__ int3 pair_delta(const PassB &a, int4 q, float lam, float2 kci, float4 rr, int4 p,
                                           const GaussPair &gpj) {
    if (GAUSS) {
        const float3 D = udiff(q, p);
        return gauss_delta(D, dot3x(D, D), lam, PACKED ? gpj : gauss_pair(kci.x, kci.y));
    }
    float3 g;
    {
        KConst c;
        c.ivd = rr.y;
        c.norm = rr.z;
        const float3 d = fdiff(q, p);
        const float r2 = dot3x(d, d);
        g = kernel_gradient(a.gk, d, r2, rr.w, c, a.gk == 1 ? gauss_height(r2, c) : 0.0f);
    }
    const float sc = lam * APBF_FIX;
    return make_int3(f2i(g.x * sc), f2i(g.y * sc), f2i(g.z * sc));
}

// Sum over particle j's row of the neighbours' terms (incompressibility_3.comp:62-66
// as a gather) and the deferred boundariness filter over the row's first fcnt
// entries.  PACKED: the neighbours' packed records (position, applied lambda) with
// j's own Gauss constants cj (every width equal); GAUSS otherwise: the packed
// records and the neighbours' Gauss constants; other kernels: the solve records
// and the positions.
template <bool GAUSS, int L, bool PACKED>
__device__ __forceinline__ int3 delta_row(const PassB &a, const int4 *pos, const uint32_t *row, uint32_t cnt,
                                          uint32_t fcnt, uint32_t j, uint32_t sub, int4 p, const GaussPair &cj,
                                          bool fil, float3 ed, bool &hit, int4 start) {
    int32_t ax = start.x, ay = start.y, az = start.z;
    // software-pipelined as in density_one: the gathers of a batch go out with the
    // row entries of the next
    // Entries are masked to their index bits: rows the search tuner leaves behind may be
    // correction rows read as transposed ones (flag bit 31), and no entry may address
    // beyond the lists (the index bits of every valid entry are the entry itself).
    uint32_t ii[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
        const uint32_t k = sub + u * L;
        ii[u] = k < cnt ? row[(size_t)k * a.stride] & ~kNoDelta : j;
    }
    for (uint32_t k0 = sub; k0 < cnt; k0 += L * kUnroll) {
        float4 rr[kUnroll];
        int4 qq[kUnroll];
        float2 kk[kUnroll];
        uint32_t in_[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            if (PACKED) {
                qq[u] = a.pk[ii[u]];
            } else if (GAUSS) {
                qq[u] = a.pk[ii[u]];
                kk[u] = a.kc[ii[u]];
            } else {
                rr[u] = a.rec[ii[u]];
                qq[u] = pos[ii[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const uint32_t k = k0 + (L * kUnroll) + u * L;
            in_[u] = k < cnt ? row[(size_t)k * a.stride] & ~kNoDelta : j;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const float lam = k0 + u * L < cnt ? (PACKED || GAUSS ? __int_as_float(qq[u].w) : rr[u].x) : 0.0f;
            int3 t;
            if (GAUSS) {
                // the deferred filter (Gauss only) shares the offset and its square with the term
                const bool ftest = fil && !hit && k0 + u * L < fcnt;
                if (lam == 0.0f && !ftest) continue;
                const float3 D = udiff(qq[u], p);
                const float r2 = dot3x(D, D);
                if (ftest) hit = gauss_filter_hit_fixed(ed, D, r2);
                if (lam == 0.0f) continue;  // the applied lambda (incompressibility_3.comp:63); padding lanes
                t = gauss_delta(D, r2, lam, PACKED ? cj : gauss_pair(kk[u].x, kk[u].y));
            } else {
                if (lam == 0.0f) continue;
                t = pair_delta<false, false>(a, qq[u], lam, kk[u], rr[u], p, cj);
            }
            ax = wadd(ax, t.x);
            ay = wadd(ay, t.y);
            az = wadd(az, t.z);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) ii[u] = in_[u];
    }
    return make_int3(ax, ay, az);
}

// Particle j's correction row (radii that differ, neighborhood.cu): terms of
// entries flagged kNoDelta subtracted (j holds them, their radius does not reach
// j), the others added (they hold j, j's radius does not reach them).  Lane sub of
// the group of L takes entries sub, sub + L, ...
template <bool GAUSS, int L, bool PACKED>
__device__ __forceinline__ int3 delta_corrections(const PassB &a, const int4 *pos, uint32_t m, uint32_t j,
                                                  uint32_t sub, int4 p, const GaussPair &cj, int3 acc) {
    for (uint32_t k = sub; k < m; k += L) {
        const uint32_t e = a.ridx[(size_t)k * a.stride + j];
        const uint32_t i = e & ~kNoDelta;
        float4 rr = make_float4(0.f, 0.f, 0.f, 0.f);
        int4 q;
        float2 kci = make_float2(0.f, 0.f);
        if (PACKED || GAUSS) {
            q = a.pk[i];
            if (!PACKED) kci = a.kc[i];
        } else {
            rr = a.rec[i];
            q = pos[i];
        }
        const float lam = PACKED || GAUSS ? __int_as_float(q.w) : rr.x;
        if (lam == 0.0f) continue;
        const int3 t = pair_delta<GAUSS, PACKED>(a, q, lam, kci, rr, p, cj);
        if (e & kNoDelta) {
            acc.x = wadd(acc.x, -t.x);
            acc.y = wadd(acc.y, -t.y);
            acc.z = wadd(acc.z, -t.z);
        } else {
            acc.x = wadd(acc.x, t.x);
            acc.y = wadd(acc.y, t.y);
            acc.z = wadd(acc.z, t.z);
        }
    }
    return acc;
}

// The end of a particle's position update: the boxes (nboxes > 0), the new position and
// the books of the lambda lj that this pass applied to it.
__device__ __forceinline__ void delta_store(const PassB &a, int4 *pos_out, uint32_t j, int4 out, bool hit, float rj,
                                            float lj, uint32_t nboxes) {
    if (hit) a.bness[j] = 0.0f;
    if (nboxes) out = box_push(out, rj, j, a.bmin, a.bmax, a.rot, nboxes);
    pos_out[j] = out;
    if (a.prev_mode | a.acc_mode) {
        accumulate(a.lam_prev, a.prev_mode, j, lj);
        accumulate(a.lam_acc, a.acc_mode, j, lj);
    }
}

// The rest of a particle's position update once its row is summed (one thread).
__device__ __forceinline__ void delta_finish(const PassB &a, int4 *pos_out, uint32_t j, int4 p, int3 acc, bool hit,
                                             float rj, float lj, uint32_t nboxes) {
    int4 out = make_int4(wadd(p.x, acc.x), wadd(p.y, acc.y), wadd(p.z, acc.z), p.w);
    delta_store(a, pos_out, j, out, hit, rj, lj, nboxes);
}

// One particle (row j_raw, lane sub of its group of L) of a position update:
// incompressibility_3 as a gather, the deferred filter, the next iteration's box
// collision (nboxes > 0) and the lambda bookkeeping.  Every lane of the group
// must call it (group shuffles).
template <bool GAUSS, int L>
__device__ __forceinline__ void delta_one(const PassB &a, const int4 *pos, int4 *pos_out, uint32_t j_raw,
                                          uint32_t n, uint32_t sub, bool packed, bool filter, const uint32_t *cnt_arr,
                                          const uint32_t *idx_arr, bool corr, uint32_t nboxes) {
    {
        const bool valid = j_raw < n;
        const uint32_t j = valid ? j_raw : 0u;
        const int4 p = pos[j];
        // j's Gauss constants as the density pass stored them
        const float2 kcj = GAUSS ? a.kc[j] : make_float2(0.f, 0.f);
        const GaussPair cj = gauss_pair(kcj.x, kcj.y);
        int32_t ax, ay, az;
        const uint32_t cnt = valid ? cnt_arr[j] : 0u;
        const uint32_t *row = idx_arr + j;
        // the self shift (incompressibility_2.comp:106-109); w flags a deferred filter
        const int4 shj = valid ? a.shift[j] : make_int4(0, 0, 0, 0);
        float3 ed = make_float3(0.f, 0.f, 0.f);
        bool fil = false, hit = false;  // this particle's deferred filter, and whether a neighbour cleared it
        uint32_t fcnt = 0;              // the filter's entries: j's own neighbours, the row's prefix
        if (filter && shj.w != 0) {
            const int4 fj = a.filt[j];
            fil = filter_dir(fj.x, fj.y, fj.z, ed);
            fcnt = a.count[j];
        }
        // the sums start from the self shift on the first lane: wrapping integer sums
        // are order-free, and the load is in flight with the particle's other data
        const int4 sh = sub == 0 ? shj : make_int4(0, 0, 0, 0);
        const float rj = a.radius[j];
        int3 acc = packed ? delta_row<GAUSS, L, true>(a, pos, row, cnt, fcnt, j, sub, p, cj, fil, ed, hit, sh)
                          : delta_row<GAUSS, L, false>(a, pos, row, cnt, fcnt, j, sub, p, cj, fil, ed, hit, sh);
        if (corr) {  // the correction row (radii that differ): usually empty
            const uint32_t m = valid ? a.rcount[j] : 0u;
            if (m) acc = packed ? delta_corrections<GAUSS, L, true>(a, pos, m, j, sub, p, cj, acc)
                                : delta_corrections<GAUSS, L, false>(a, pos, m, j, sub, p, cj, acc);
        }
        ax = acc.x;
        ay = acc.y;
        az = acc.z;
        if (L > 1) {
            ax = group_wsum<L>(ax);
            ay = group_wsum<L>(ay);
            az = group_wsum<L>(az);
            if (filter) {
                int h = hit ? 1 : 0;
#pragma unroll
                for (int off = L / 2; off > 0; off >>= 1) h |= __shfl_xor_sync(0xffffffffu, h, off);
                hit = h != 0;
            }
        }
        if (!valid || sub != 0) return;
        // applied (learned) lambda
        const float lj = (a.prev_mode | a.acc_mode) ? __int_as_float(a.pk[j].w) : 0.0f;
        delta_finish(a, pos_out, j, p, make_int3(ax, ay, az), hit, rj, lj, nboxes);
    }
}

// A converged pass (no position update) of particle j: the deferred filter still
// belongs to it, the positions are copied through and nothing is applied.
__device__ __forceinline__ void delta_skip_filter(const PassB &a, const int4 *pos, uint32_t j) {
    if (!a.shift[j].w) return;
    const int4 fj = a.filt[j];
    float3 ed;
    if (!filter_dir(fj.x, fj.y, fj.z, ed)) return;
    const int4 p = pos[j];
    for (uint32_t k = 0; k < a.count[j]; ++k)
        if (gauss_filter_hit(ed, fdiff(p, pos[a.idx[(size_t)k * a.stride + j]]))) {
            a.bness[j] = 0.0f;
            break;
        }
}
__device__ __forceinline__ void delta_skip_copy(const PassB &a, uint32_t j) {
    a.pos_out[j] = a.pos[j];
    accumulate(a.lam_prev, a.prev_mode, j, 0.0f);  // nothing applied in this pass
    accumulate(a.lam_acc, a.acc_mode, j, 0.0f);
}

// What every block of a position update works out before its particles: the list's
// length, the row forms, whether the pass runs and, in block 0, the books of the
// density pass behind it (PassSync).  Every calling warp is whole, block 0's first among
// them.
struct UpdateHead {
    uint32_t n, nboxes;
    bool skip, filter, sym, corr, packed;
};
// The books of a pass and the slot of the next (one warp); a call, so that its few
// instructions in one block cost the others no registers.
__device__ __noinline__ void update_books(const PassB &a, uint32_t n, uint32_t slot, PassTotals t, bool ran, bool met) {
    if (threadIdx.x < (uint32_t)kSumStripes)
        for (int k = 0; k < 3; ++k) a.sync->e[slot ^ 1u][threadIdx.x][k] = 0ull;
    if (threadIdx.x != 0u) return;
    if (ran) {
        a.st->kw_uniform = t.kw_diff ? 0u : 1u;
        finish_pass(a.red_out, a.st, a.target, n, (long long)t.e1, (long long)t.e2, met);
    }
    a.sync->cur_density = slot ^ 1u;
    if (a.loop_end) {  // once more while no pass met the target and passes remain
        const uint32_t next = a.st->pass_index + 2u;
        a.st->pass_start = next;
        a.st->loop_iters += 1u;
        cudaGraphSetConditional(a.loop_handle, a.st->converged == 0u && next < a.max_passes ? 1u : 0u);
    }
}
template <bool GAUSS>
__device__ __forceinline__ UpdateHead update_head(const PassB &a, uint32_t n) {
    UpdateHead h;
    h.n = n;
    const uint32_t slot = *(volatile const uint32_t *)&a.sync->cur_update & 1u;
    h.skip = a.early_exit && *(volatile const uint32_t *)&a.st->converged;
    h.nboxes = a.nboxes;
    if (a.loop_offset >= 0) {
        const uint32_t pass = a.st->pass_index + (uint32_t)a.loop_offset;
        h.skip = h.skip || pass >= a.max_passes;
        if (pass + 1u >= a.max_passes) h.nboxes = 0u;  // no box collision after the last iteration
    }
    const PassTotals t = pass_totals(a.sync, slot);
    // every block decides for itself from the sums: block 0 may be setting the flag of
    // this pass, and reading it early or late gives the same answer
    const bool ran = !h.skip;
    if (ran && a.early_exit) h.skip = error_meets_target(t.e1, n, a.target, a.target_m, a.target_s);
    if (blockIdx.x == 0 && threadIdx.x < 32u) update_books(a, n, slot, t, ran, h.skip);
    // the density pass of this pass deferred the Gauss filter to here (symmetric rows)
    h.filter = GAUSS && *(volatile const uint32_t *)&a.st->filter_tag != 0u;
    // Rows: symmetric (equal radii) or with correction rows (the green search with
    // radii that differ): the particle's own row; transposed rows otherwise.
    h.sym = a.st->range_min == a.st->range_max;
    h.corr = !h.sym && a.st->union_rows != 0u;
    // Equal kernel widths (same bits): every neighbour's Gauss constants are this
    // particle's, so one 16-byte record (position, applied lambda) per neighbour is
    // gathered instead of the solve record and the position.
    h.packed = GAUSS && !t.kw_diff;
    return h;
}
// A converged pass: no position update, but its deferred filter still runs.
__device__ __forceinline__ void update_skipped(const PassB &a, const UpdateHead &h) {
    if (h.filter)
        for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < h.n; j += gridDim.x * blockDim.x)
            delta_skip_filter(a, a.pos, j);
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < h.n; j += gridDim.x * blockDim.x)
        delta_skip_copy(a, j);
}

template <bool GAUSS, int L>
__global__ void __launch_bounds__(256, 4) k_delta(PassB a) {
    grid_dependency_wait();
    grid_dependency_trigger();
    const UpdateHead h = update_head<GAUSS>(a, a.d_len[kLenParticles]);
    if (h.skip) {
        update_skipped(a, h);
        return;
    }
    const uint32_t *cnt_arr = h.sym || h.corr ? a.count : a.rcount;
    const uint32_t *idx_arr = h.sym || h.corr ? a.idx : a.ridx;
    const uint32_t sub = threadIdx.x % L;
    const uint32_t gpb = blockDim.x / L;
    for (uint32_t base = blockIdx.x * gpb; base < h.n; base += gridDim.x * gpb)
        delta_one<GAUSS, L>(a, a.pos, a.pos_out, base + threadIdx.x / L, h.n, sub, h.packed, h.filter, cnt_arr, idx_arr,
                            h.corr, h.nboxes);
}

// ---- the two passes over tiles of particles ----
//
// The direct passes above gather a 16-byte record per pair.  Their warps wait for
// those gathers (42 % of them leave the L1 at a million particles) and idle a third of
// their lanes, because neighbouring particles have rows of different lengths.  The rows
// of a substep do not change between its passes, so for the solve they are rewritten
// once (k_tile_rows): T consecutive particles are a tile, the particles outside it
// that its rows name are its halo (1.6 per particle at T = 128, against 14 to 22 row
// entries), row entries become 16-bit byte offsets of records (the tile's T, T null
// records that pad odd rows, the halo's), and the tile's particles are dealt to its
// threads by falling row length.  A pass then loads a
// tile's records into shared memory once, with every load in flight together, and
// its pair loop reads shared memory only.  The pair arithmetic and the integer sums are
// the direct passes' own, so the results are bit-identical.
//
// Entries from kTileDepth on and tiles whose halo exceeds kTileHalo are read from the list's
// own rows, or from the pool (rests_by_lane).

// Eight neighbouring particles, whose records share a line, keep together in the table and
// so in the halo, which takes its order; the groups are spread.  A group that finds its eight
// slots taken looks at the next eight, so that its keys take a step each and not eight (a tile
// of many outside particles 68 -> 28 us, all tiles of a drop of 250 000 42 -> 35).
__device__ __forceinline__ uint32_t tile_hash(uint32_t j, uint32_t mask) {
    return (((j >> 3) * 2654435761u >> 16) << 3 | (j & 7u)) & mask;
}

// Who walks the entries from kTileDepth on of a tile's `rows` long rows, `longest` entries
// the longest: their own threads (true), a memory latency for every four entries but all
// rows at once, or each row a whole warp, two latencies for every 128 entries and the sums
// across it, one row after the other.  Rows are dealt by falling length, so a tile's long
// ones share warps.  Whole warps alone took 2.1 times the direct passes' time where all rows
// are long (512 000 particles with rows of 181 entries, eight passes: 13.9 against 6.5 ms).
__device__ __forceinline__ bool rests_by_lane(uint32_t rows, uint32_t longest) {
    const uint32_t rest = longest - (uint32_t)kTileDepth;
    return rows >= 32u || (rows != 0u && rows * (2u * (rest / 128u) + 3u) > rest);
}

struct TileRowsArgs {
    const uint32_t *count, *idx;
    uint32_t stride;
    const float *radius;
    const uint32_t *d_len;
    const Status *st;
    int reverse;  // transposed rows: needed when neither symmetric nor correction rows hold
    TilePlan plan;
};

template <int T>
__global__ void __launch_bounds__(256) k_tile_rows(TileRowsArgs a) {
    constexpr uint32_t S = 256 / T;    // threads per particle
    constexpr uint32_t kSlots = 2048;  // hash table, at most 32 % full
    constexpr uint32_t kProbes = 64;   // slots looked at before a tile counts as overflowing
    constexpr uint32_t kKept = 8;      // row quads whose table slots are kept from the first walk
    static_assert(kTileHalo * 2 <= kSlots, "the hash table holds the halo with room to probe");
    __shared__ uint32_t s_key[kSlots];
    __shared__ uint16_t s_val[kSlots];
    __shared__ uint2 s_kept[kKept * T];  // four 16-bit codes: 0x8000 | table slot, or the offset of a tile record
    __shared__ uint32_t s_bin[64];
    __shared__ uint16_t s_rank[T];
    __shared__ uint32_t s_scan[8];
    __shared__ uint32_t s_full, s_rmax, s_long, s_longest;
    if (a.reverse && (a.st->range_min == a.st->range_max || a.st->union_rows != 0u)) return;
    const uint32_t n = a.d_len[kLenParticles];
    const uint32_t o = threadIdx.x % T, sub = threadIdx.x / T;  // a warp reads consecutive particles' entries
    for (uint32_t tile = blockIdx.x; tile * T < n; tile += gridDim.x) {
        const uint32_t base = tile * T, i = base + o;
        const uint32_t cnt = i < n ? a.count[i] : 0u;
        const float r = i < n ? fabsf(a.radius[i]) : 0.0f;
        for (uint32_t k = threadIdx.x; k < kSlots; k += 256) s_key[k] = 0xffffffffu;
        if (threadIdx.x < 64) s_bin[threadIdx.x] = 0u;
        if (threadIdx.x == 0) s_full = s_rmax = s_long = s_longest = 0u;
        __syncthreads();
        const uint32_t depth = min(cnt, (uint32_t)kTileDepth);
        // falling row length: a counting sort (the order among equal lengths is free)
        const uint32_t bin = 63u - min(cnt, 63u);
        if (sub == 0) atomicAdd(&s_bin[bin], 1u);
        const uint32_t rm = __reduce_max_sync(0xffffffffu, __float_as_uint(r));
        if ((threadIdx.x & 31u) == 0u) atomicMax(&s_rmax, rm);
        if (sub == 0) {
            const uint32_t lm = __ballot_sync(0xffffffffu, cnt > kTileDepth), most = __reduce_max_sync(0xffffffffu, cnt);
            if (lm && (threadIdx.x & 31u) == 0u) {
                atomicAdd(&s_long, (uint32_t)__popc(lm));
                atomicMax(&s_longest, most);
            }
        }
        // the code of entry j: the offset of its record when it lies in the tile, else
        // its slot in the table of the halo, entered when it is not there yet.  Only the keys
        // are entered here; numbering them here as well (a counter that every insert waits
        // for) made this walk four fifths of the kernel.
        const auto enter = [&](uint32_t j) -> uint32_t {
            if (j - base < T) return (j - base) * 16u;
            uint32_t h = tile_hash(j, kSlots - 1);
            for (uint32_t probe = 0; probe < kProbes; ++probe) {
                uint32_t was = *(volatile uint32_t *)&s_key[h];
                if (was == 0xffffffffu) was = atomicCAS(&s_key[h], 0xffffffffu, j);
                if (was == j || was == 0xffffffffu) return 0x8000u | h;
                h = (h + 8u) & (kSlots - 1);
            }
            s_full = 1u;  // far more outside particles than the halo holds
            return 0u;
        };
        const auto load4 = [&](uint32_t q, uint32_t (&j)[4]) {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) j[u] = 4u * q + u < depth ? a.idx[(size_t)(4u * q + u) * a.stride + i] : i;
        };
        uint32_t j[4];
        load4(sub, j);
#pragma unroll 1
        for (uint32_t q = sub; 4u * q < depth; q += S) {
            uint32_t nx[4];
            load4(q + S, nx);
            uint32_t c[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) c[u] = 4u * q + u < depth ? enter(j[u]) : (T + o) * 16u;
            if (q < kKept) s_kept[q * T + o] = make_uint2(c[0] | c[1] << 16, c[2] | c[3] << 16);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) j[u] = nx[u];
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // exclusive scan of the 64 bins
            const uint32_t x0 = s_bin[2 * threadIdx.x], x1 = s_bin[2 * threadIdx.x + 1];
            uint32_t v = x0 + x1;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, v, off);
                if ((int)threadIdx.x >= off) v += y;
            }
            s_bin[2 * threadIdx.x] = v - x0 - x1;
            s_bin[2 * threadIdx.x + 1] = v - x1;
        }
        // the halo in the table's order: a thread numbers the keys of eight slots
        constexpr uint32_t kPer = kSlots / 256;
        uint32_t key[kPer], used = 0;
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) {
            key[u] = s_key[threadIdx.x * kPer + u];
            used += key[u] != 0xffffffffu ? 1u : 0u;
        }
        uint32_t first = used;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, first, off);
            if ((int)(threadIdx.x & 31u) >= off) first += y;
        }
        if ((threadIdx.x & 31u) == 31u) s_scan[threadIdx.x / 32u] = first;
        __syncthreads();
        uint32_t halo = 0;
        first -= used;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
            const uint32_t c = s_scan[w];
            if (w < threadIdx.x / 32u) first += c;
            halo += c;
        }
        const bool over = halo > kTileHalo || s_full != 0u;
        if (!over) {
#pragma unroll
            for (uint32_t u = 0; u < kPer; ++u) {
                if (key[u] == 0xffffffffu) continue;
                s_val[threadIdx.x * kPer + u] = (uint16_t)((2 * T + first) * 16u);
                a.plan.halo[(size_t)tile * kTileHalo + first] = key[u];
                ++first;
            }
        }
        if (sub == 0) {
            const uint32_t k = atomicAdd(&s_bin[bin], 1u);
            s_rank[o] = (uint16_t)k;
            a.plan.lane[base + k] = i < n ? o | cnt << 8 : kNoParticle;
        }
        // the rest of the long rows, each in one run of the pool: read through the list's
        // own rows by a warp, every entry would touch another page
        const bool lanes = rests_by_lane(s_long, s_longest);
        if (sub == 0 && !lanes)
            for (uint32_t left = __ballot_sync(0xffffffffu, cnt > kTileDepth); left; left &= left - 1u) {
                const int src = __ffs(left) - 1;
                const uint32_t li = __shfl_sync(0xffffffffu, i, src), m = __shfl_sync(0xffffffffu, cnt, src) - kTileDepth;
                const uint32_t lane = threadIdx.x & 31u;
                uint32_t at = 0;
                if ((int)lane == src) {
                    at = pool_run(atomicAdd(a.plan.pool_used, (PoolCount)m), m, a.plan.pool_size);
                    a.plan.tail[i] = at;
                }
                at = __shfl_sync(0xffffffffu, at, src);
                if (at != kNoRun)
                    for (uint32_t k = lane; k < m; k += 32u)
                        a.plan.pool[at + k] = a.idx[(size_t)(kTileDepth + k) * a.stride + li];
            }
        if (threadIdx.x == 0)
            a.plan.tile[tile] = make_uint4(over ? kHaloOver : halo, min(n - base, (uint32_t)T), s_rmax, lanes ? 1u : 0u);
        __syncthreads();
        if (!over) {
            uint2 *out = a.plan.rows + (size_t)tile * (T * kTileDepth / 4) + s_rank[o];
            const auto offset = [&](uint32_t c) { return c & 0x8000u ? (uint32_t)s_val[c & 0x7fffu] : c; };
#pragma unroll 1
            for (uint32_t q = sub; q * 4u < depth; q += S) {
                uint32_t c[4];
                if (q < kKept) {
                    const uint2 k = s_kept[q * T + o];
                    c[0] = k.x & 0xffffu;
                    c[1] = k.x >> 16;
                    c[2] = k.y & 0xffffu;
                    c[3] = k.y >> 16;
                } else {
                    load4(q, j);
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) c[u] = 4u * q + u < depth ? enter(j[u]) : (T + o) * 16u;
                }
                out[q * T] =
                    make_uint2(offset(c[0]) | offset(c[1]) << 16, offset(c[2]) | offset(c[3]) << 16);
            }
        }
        __syncthreads();  // the shared arrays are the next tile's
    }
}

// Two FP32 values in one 64-bit register pair: the packed operations round each half
// like the scalar ones, at half the issue slots.  A packed product followed by a packed sum
// gave the values of one FMA, whatever the rounding modifiers and -fmad, where the passes
// must round twice (dot3x): sums are written as fma(a, 1, b), which rounds a + b once, with
// the 1 taken from the kernel's arguments so that it stays a value.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2_pack(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b, F2 one) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(one.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 dot3_f2(F2 ax, F2 ay, F2 az, F2 bx, F2 by, F2 bz, F2 one) {
    return f2_add(f2_add(ax * bx, ay * by, one), az * bz, one);
}
__device__ __forceinline__ float ex2_ftz(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The Gauss height W and the gradient factor s (gradient = s D) of two offsets at
// once, as gauss_terms_r2 computes them, for exponents of at least -126: 2^-126 is the
// smallest normal number, so down to there ex2_ftz flushes nothing, and its values are exp2f's
// (test_gpu_exponential.py compares all of them).  low collects the smallest exponent; a row
// in which it fell below is summed again by gauss_terms_r2.
__device__ __forceinline__ void gauss_two(F2 r2, F2 ivd36, F2 norm, F2 k2, float &low, F2 &W, F2 &s) {
    const float2 x = f2_unpack(r2 * ivd36);
    low = fminf(fminf(low, x.x), x.y);
    W = f2_pack(ex2_ftz(x.x), ex2_ftz(x.y)) * norm;
    const float2 t = f2_unpack(W * k2), q = f2_unpack(r2);
    // no gradient below 0.0001 reference units
    s = f2_pack(q.x < 1.0e-8f * 0x1p36f ? 0.0f : t.x, q.y < 1.0e-8f * 0x1p36f ? 0.0f : t.y);
}
constexpr float kLowExponent = -126.0f;

__device__ __forceinline__ const int4 &tile_record(const int4 *s_rec, uint32_t offset) {
    return *reinterpret_cast<const int4 *>(reinterpret_cast<const char *>(s_rec) + offset);
}
__device__ __forceinline__ uint32_t row_offset(uint2 e, uint32_t u) {
    const uint32_t w = (u & 2u) ? e.y : e.x;
    return (u & 1u) ? w >> 16 : w & 0xffffu;
}

// Exact sum over a warp of 32-bit values, as two 16-bit halves.
__device__ __forceinline__ long long warp_sum32(int32_t v) {
    const int32_t hi = __reduce_add_sync(0xffffffffu, v >> 16);
    const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0xffffu);
    return ((long long)hi << 16) + (long long)lo;
}

// The entries from kTileDepth on of lane src's row, walked by its whole warp: lane l takes
// entries l, l + 32, ... of them, four loads in flight.  A lane alone would wait two memory
// latencies for every entry.
struct WarpRow {
    const uint32_t *entry;
    size_t stride;
    uint32_t m;
    int4 p;
    __device__ __forceinline__ WarpRow(const TilePlan &plan, const uint32_t *idx, uint32_t row_stride, uint32_t i_,
                                       uint32_t cnt_, const int4 &p_, int src) {
        const uint32_t i = __shfl_sync(0xffffffffu, i_, src);
        m = __shfl_sync(0xffffffffu, cnt_, src) - kTileDepth;
        p.x = __shfl_sync(0xffffffffu, p_.x, src);
        p.y = __shfl_sync(0xffffffffu, p_.y, src);
        p.z = __shfl_sync(0xffffffffu, p_.z, src);
        p.w = 0;
        const uint32_t at = plan.tail[i];
        entry = at != kNoRun ? plan.pool + at : idx + (size_t)kTileDepth * row_stride + i;
        stride = at != kNoRun ? 1u : row_stride;
    }
    template <typename G, typename F>
    __device__ __forceinline__ void each(G load, F f) const {
        for (uint32_t k0 = threadIdx.x & 31u; k0 < m; k0 += 128u) {
            uint32_t j[4];
            int4 q[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) j[u] = k0 + 32u * u < m ? entry[(k0 + 32u * u) * stride] : 0u;
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) q[u] = k0 + 32u * u < m ? load(j[u]) : make_int4(0, 0, 0, 0);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if (k0 + 32u * u < m) f(j[u], q[u]);
        }
    }
};

// Entries k, k + L, ... below end of a list's row, walked by one thread: four gathers (`load`)
// in flight with the four entries behind them.
template <uint32_t L, typename G, typename F>
__device__ __forceinline__ void lane_row(const uint32_t *row, size_t stride, uint32_t k, uint32_t end, G load, F f) {
    if (k >= end) return;
    uint32_t j[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u) j[u] = k + u * L < end ? row[(k + u * L) * stride] : 0u;
#pragma unroll 1
    for (; k < end; k += 4u * L) {
        decltype(load(0u)) q[4];
        uint32_t nj[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) q[u] = load(j[u]);
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) nj[u] = k + (4u + u) * L < end ? row[(k + (4u + u) * L) * stride] : 0u;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (k + u * L < end) f(q[u]);
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) j[u] = nj[u];
    }
}

// A tile's density pass: T particles, L threads each.  At a million particles in a
// waterfall (13.4 M pairs) 55 us against 96 us for the direct kernel, 25 against 35 us at
// 250 000 (4.45 M pairs).  Bound by the latency of a tile's own loads (three rounds: the
// plan's words, the records, the barrier): half of a block's time, while the pair loop
// issues at 55 % of the cycles; so the plan's words come in one round and before the
// kernel in front has ended, and eight blocks (64 registers) share an SM.
template <int T, int L>
__global__ void __launch_bounds__(T *L, 1024 / (T * L)) k_density_tiles(PassA a, TilePlan plan) {
    extern __shared__ int4 s_pos[];  // the tile's records, its null records, its halo's; w: mass x 2^18
    constexpr uint32_t B = T * L;
    const uint32_t n = a.d_len[kLenParticles];
    const uint32_t sub = threadIdx.x % L, rank = threadIdx.x / L;
    bool defer = false;
    uint32_t slot = 0;
    PassSums ps;
    for (uint32_t tile = blockIdx.x; tile * T < n || tile == 0u; tile += gridDim.x) {
        // what stays between the passes of a substep first, in one round of loads (those
        // beyond the tile's row lengths and halo are not used): with a programmatic launch
        // they run while the kernel before drains
        const uint32_t base = tile * T;
        const uint4 head = plan.tile[tile];
        const uint32_t lane = plan.lane[base + rank];
        const uint2 *row = plan.rows + (size_t)tile * (T * kTileDepth / 4) + rank;
        const uint32_t *halo = plan.halo + (size_t)tile * kTileHalo;
        const uint32_t h0 = halo[threadIdx.x], h1 = halo[threadIdx.x + B];
        uint2 e = row[sub * T];
        if (tile == blockIdx.x) grid_dependency_trigger();
        const bool over = head.x == kHaloOver;
        const uint32_t H = over || n == 0u ? 0u : head.x;
        const bool valid = n != 0u && lane != kNoParticle;
        const uint32_t o = valid ? lane & 255u : 0u, i = base + o;
        const uint32_t cnt = valid ? lane >> 8 : 0u;
        const float kw = a.kw[i], im = a.inv_mass[i], radius = a.radius[i];
        ps.kw0 = __float_as_uint(a.kw[0]);
        const uint32_t depth = over ? 0u : min(cnt, (uint32_t)kTileDepth);
        if (tile == blockIdx.x) {
            grid_dependency_wait();
            const bool skip = (a.early_exit && *(volatile uint32_t *)&a.st->converged) || loop_over(a);
            defer = a.filt && a.method == 2 && (a.st->range_min == a.st->range_max || a.st->union_rows != 0u);
            slot = *(volatile uint32_t *)&a.sync->cur_density & 1u;
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                a.st->filter_tag = (!skip && defer) ? 1u : 0u;
                a.sync->cur_update = slot;
                a.sync->pool_used[0] = a.sync->pool_used[1] = 0ull;  // for the next substep's rows
            }
            if (skip || n == 0u) return;  // uniform over the grid
        }
        const auto stage = [&](uint32_t k, uint32_t g) {
            int4 v = a.pos[g];
            v.w = __float_as_int(__int_as_float(v.w) * APBF_FIX);
            s_pos[k] = v;
        };
        const float b0 = a.bness[i], pushed = a.projected ? a.lam_prev[i] : 0.0f;
        for (uint32_t k = threadIdx.x; k < T; k += B)
            if (k < head.y) {
                const int4 v = a.pos[base + k];
                s_pos[k] = make_int4(v.x, v.y, v.z, __float_as_int(__int_as_float(v.w) * APBF_FIX));
                s_pos[T + k] = make_int4(v.x, v.y, v.z, 0);
            }
        if (threadIdx.x < H) stage(2 * T + threadIdx.x, h0);
        if (threadIdx.x + B < H) stage(2 * T + B + threadIdx.x, h1);
        for (uint32_t k = threadIdx.x + 2 * B; k < H; k += B) stage(2 * T + k, halo[k]);
        __syncthreads();
        const int4 p = s_pos[o];
        const KConst c = gauss_consts(kw);
        const GaussPair gp = gauss_pair(c);
        RowSums rs;
        float low = 0.0f;
        {
            const F2 one = f2_pack(a.one, a.one);
            const F2 ivd = f2_pack(gp.ivd36, gp.ivd36), norm = f2_pack(gp.norm, gp.norm), kk = f2_pack(gp.k2, gp.k2);
            const auto two = [&](uint32_t w) {
                const int4 q0 = tile_record(s_pos, w & 0xffffu), q1 = tile_record(s_pos, w >> 16);
                const F2 dx = f2_pack((float)wadd(q0.x, -p.x), (float)wadd(q1.x, -p.x));
                const F2 dy = f2_pack((float)wadd(q0.y, -p.y), (float)wadd(q1.y, -p.y));
                const F2 dz = f2_pack((float)wadd(q0.z, -p.z), (float)wadd(q1.z, -p.z));
                const F2 m = f2_pack(__int_as_float(q0.w), __int_as_float(q1.w));
                F2 W, s;
                gauss_two(dot3_f2(dx, dy, dz, dx, dy, dz, one), ivd, norm, kk, low, W, s);
                const F2 gx = s * dx, gy = s * dy, gz = s * dz;
                const float2 tw = f2_unpack(W * m), tx = f2_unpack(gx * m), ty = f2_unpack(gy * m),
                             tz = f2_unpack(gz * m), tq = f2_unpack(dot3_f2(gx, gy, gz, gx, gy, gz, one) * m);
                rs.dens += f2u(tw.x) + f2u(tw.y);
                rs.gx = wadd(rs.gx, wadd(f2i(tx.x), f2i(tx.y)));
                rs.gy = wadd(rs.gy, wadd(f2i(ty.x), f2i(ty.y)));
                rs.gz = wadd(rs.gz, wadd(f2i(tz.x), f2i(tz.y)));
                rs.sq += f2u(tq.x) + f2u(tq.y);
            };
            for (uint32_t k = sub * 4u; k < depth; k += L * 4u) {
                const uint2 cur = e;
                if (k + L * 4u < depth) e = row[(k / 4u + L) * T];
                two(cur.x);
                if (k + 2u < depth) two(cur.y);
            }
        }
        const auto add = [&](int4 q, float mjf) {
            float W;
            float3 g;
            gauss_terms(udiff(p, q), gp, W, g);
            rs.dens += f2u(W * mjf);
            rs.gx = wadd(rs.gx, f2i(g.x * mjf));
            rs.gy = wadd(rs.gy, f2i(g.y * mjf));
            rs.gz = wadd(rs.gz, f2i(g.z * mjf));
            rs.sq += f2u(dot3x(g, g) * mjf);
        };
        if (L > 1) low = group_min<L>(low);  // the group sums its row again as one
        if (low < kLowExponent) {  // far out in a narrow kernel: subnormal results
            rs = RowSums();
#pragma unroll 1
            for (uint32_t k = sub; k < depth; k += L) {
                const int4 q = tile_record(s_pos, row_offset(row[(k / 4u) * T], k));
                add(q, __int_as_float(q.w));
            }
        }
        // what the tile does not hold: all of the rows where its halo did not fit, and the rest
        // of the long ones, by their threads or one row after the other by the whole warp
        const bool by_warp = head.w == 0u && cnt > kTileDepth;
        const uint32_t end = by_warp ? (uint32_t)kTileDepth : cnt;
        lane_row<L>(a.idx + i, a.stride, depth + sub, end, [&](uint32_t j) { return a.pos[j]; },
                    [&](const int4 &q) { add(q, __int_as_float(q.w) * APBF_FIX); });
        for (uint32_t left = __ballot_sync(0xffffffffu, sub == 0u && by_warp); left; left &= left - 1u) {
            const int src = __ffs(left) - 1;
            const WarpRow w(plan, a.idx, a.stride, i, cnt, p, src);
            const GaussPair gw = gauss_pair(__shfl_sync(0xffffffffu, gp.ivd36, src), __shfl_sync(0xffffffffu, gp.norm, src));
            RowSums t;
            w.each([&](uint32_t j) { return a.pos[j]; }, [&](uint32_t, const int4 &q) {
                const float mjf = __int_as_float(q.w) * APBF_FIX;
                float W;
                float3 g;
                gauss_terms(udiff(w.p, q), gw, W, g);
                t.dens += f2u(W * mjf);
                t.gx = wadd(t.gx, f2i(g.x * mjf));
                t.gy = wadd(t.gy, f2i(g.y * mjf));
                t.gz = wadd(t.gz, f2i(g.z * mjf));
                t.sq += f2u(dot3x(g, g) * mjf);
            });
            const uint32_t d = __reduce_add_sync(0xffffffffu, t.dens), s2 = __reduce_add_sync(0xffffffffu, t.sq);
            const int32_t x = __reduce_add_sync(0xffffffffu, t.gx), y = __reduce_add_sync(0xffffffffu, t.gy),
                          z = __reduce_add_sync(0xffffffffu, t.gz);
            if ((int)(threadIdx.x & 31u) == src) {
                rs.dens += d;
                rs.sq += s2;
                rs.gx = wadd(rs.gx, x);
                rs.gy = wadd(rs.gy, y);
                rs.gz = wadd(rs.gz, z);
            }
        }
        if (L > 1) {
            rs.dens = group_sum<L>(rs.dens);
            rs.sq = group_sum<L>(rs.sq);
            rs.gx = group_wsum<L>(rs.gx);
            rs.gy = group_wsum<L>(rs.gy);
            rs.gz = group_wsum<L>(rs.gz);
        }
        PassSums one;
        one.kw0 = ps.kw0;
        float3 ed = make_float3(0.f, 0.f, 0.f);
        bool ask = false;
        if (valid && sub == 0)
            ask = density_finish<true, false>(a, a.pos, i, make_int4(p.x, p.y, p.z, 0), kw, c, gp, cnt, rs, im, radius, b0,
                                              pushed, false, defer, false, one, ed);
        if (__any_sync(0xffffffffu, ask)) {  // the boundariness filter of transposed rows
            bool hit = false;
            if (ask) {
                uint2 r = depth ? row[0] : make_uint2(0u, 0u);
#pragma unroll 1
                for (uint32_t k = 0; k < depth && !hit; k += 4u) {  // (a null record never hits)
                    const uint2 now = r;
                    if (k + 4u < depth) r = row[(k / 4u + 1u) * T];
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u)
                        hit = hit || gauss_filter_hit(ed, fdiff(p, tile_record(s_pos, row_offset(now, u))));
                }
#pragma unroll 2
                for (uint32_t k = depth; k < end && !hit; ++k)
                    hit = gauss_filter_hit(ed, fdiff(p, a.pos[a.idx[(size_t)k * a.stride + i]]));
            }
            for (uint32_t left = __ballot_sync(0xffffffffu, ask && !hit && by_warp); left; left &= left - 1u) {
                const int src = __ffs(left) - 1;
                const WarpRow w(plan, a.idx, a.stride, i, cnt, p, src);
                const float3 ew = make_float3(__shfl_sync(0xffffffffu, ed.x, src), __shfl_sync(0xffffffffu, ed.y, src),
                                              __shfl_sync(0xffffffffu, ed.z, src));
                bool any = false;
                w.each([&](uint32_t j) { return a.pos[j]; },
                       [&](uint32_t, const int4 &q) { any = any || gauss_filter_hit(ew, fdiff(w.p, q)); });
                any = __any_sync(0xffffffffu, any);
                if ((int)(threadIdx.x & 31u) == src) hit = any;
            }
            if (hit) a.bness[i] = 0.0f;
        }
        ps.e1 += warp_sum32((int32_t)one.e1);  // one term each, in 32 bits (err_fix)
        ps.e2 += warp_sum32((int32_t)one.e2);
        ps.kw_diff = ps.kw_diff || one.kw_diff;
        if (tile + gridDim.x < (n + T - 1) / T) __syncthreads();  // the shared records are the next tile's
    }
    __shared__ long long s_e[2][B / 32];
    if ((threadIdx.x & 31u) == 0u) {
        s_e[0][threadIdx.x / 32u] = ps.e1;
        s_e[1][threadIdx.x / 32u] = ps.e2;
    }
    PassSums bs;
    bs.kw_diff = __syncthreads_or(ps.kw_diff) != 0;
    if (threadIdx.x == 0) {
        for (uint32_t k = 0; k < B / 32u; ++k) {
            bs.e1 += s_e[0][k];
            bs.e2 += s_e[1][k];
        }
        add_pass_sums(a.sync, slot, bs);
    }
}

// Boxes that can move no particle of a tile.  Thread k writes box k's outer faces for the
// tile's largest |radius|: box_clear's own thresholds, which only move outwards as the
// radius grows (rounding is monotone), so a position outside them is outside the
// particle's.  Per box: the faces (w of the first word: 0 axis-aligned, 1 oriented, 2 beyond
// box_clear's range, then the box itself is asked), the rotation's rows, the centre.
constexpr uint32_t kTileBoxes = 8, kTileBoxWords = 6;
__device__ __forceinline__ void tile_box(const PassB &a, uint32_t k, float rmax, float4 *s_box) {
    const float c = 0.0500001f;
    const float4 lo = a.bmin[k], hi = a.bmax[k], r0 = a.rot[3 * k];
    const bool oriented = r0.w != 0.0f;
    const float3 l = oriented ? make_float3(-hi.x, -hi.y, -hi.z) : make_float3(lo.x, lo.y, lo.z);
    const float4 b0 = make_float4(__fsub_rn(__fsub_rn(l.x, rmax), c), __fsub_rn(__fsub_rn(l.y, rmax), c),
                                  __fsub_rn(__fsub_rn(l.z, rmax), c), 0.0f);
    const float4 b1 = make_float4(__fadd_rn(__fadd_rn(hi.x, rmax), c), __fadd_rn(__fadd_rn(hi.y, rmax), c),
                                  __fadd_rn(__fadd_rn(hi.z, rmax), c), 0.0f);
    const float m = fmaxf(fmaxf(fmaxf(fabsf(b0.x), fabsf(b0.y)), fmaxf(fabsf(b0.z), fabsf(b1.x))),
                          fmaxf(fabsf(b1.y), fabsf(b1.z)));
    float4 *w = s_box + kTileBoxWords * k;
    w[0] = make_float4(b0.x, b0.y, b0.z, !(m < 1.0e30f) ? 2.0f : (oriented ? 1.0f : 0.0f));
    w[1] = b1;
    if (oriented) {
        w[2] = r0;
        w[3] = a.rot[3 * k + 1];
        w[4] = a.rot[3 * k + 2];
        w[5] = lo;
    }
}
// The first box that may push v (nb: none).
__device__ __forceinline__ uint32_t tile_boxes_clear(int4 v, const float4 *s_box, uint32_t nb) {
    const float px = __fmul_rn((float)v.x, 0x1p-18f), py = __fmul_rn((float)v.y, 0x1p-18f),
                pz = __fmul_rn((float)v.z, 0x1p-18f);
    uint32_t first = nb;
#pragma unroll 1
    for (uint32_t k = nb; k-- > 0u;) {
        const float4 *w = s_box + kTileBoxWords * k;
        const float4 b0 = w[0], b1 = w[1];
        float qx = px, qy = py, qz = pz;
        if (b0.w != 0.0f) {  // as box_push takes the position into the box's frame
            const float4 c = w[5];
            const float dx = __fsub_rn(px, c.x), dy = __fsub_rn(py, c.y), dz = __fsub_rn(pz, c.z);
            qx = dot3_rn(w[2], dx, dy, dz);
            qy = dot3_rn(w[3], dx, dy, dz);
            qz = dot3_rn(w[4], dx, dy, dz);
        }
        const bool clear = b0.w != 2.0f && (qx < b0.x || qy < b0.y || qz < b0.z || qx >= b1.x || qy >= b1.y || qz >= b1.z);
        if (!clear) first = k;
    }
    return first;
}
// box_push from box `first` on, where the boxes before it are known to leave ip alone.
__device__ __noinline__ int4 box_push_from(int4 ip, float r, uint32_t id, const float4 *__restrict__ bmin,
                                           const float4 *__restrict__ bmax, const float4 *__restrict__ rot,
                                           uint32_t first, uint32_t nb) {
    return box_push(ip, r, id, bmin + first, bmax + first, rot + 3 * first, nb - first);
}

// A tile's position update.  fwd: the plan of the own rows, rev: that of the
// transposed rows.  79 us at a million particles against 127 us for the direct kernel, 29
// against 37 us at 250 000.  Of its instructions the deferred filter's row tests took a
// quarter and the boxes a fifth; both now reject by cheap bounds first.
template <int T, int L>
__global__ void __launch_bounds__(T *L, 896 / (T * L)) k_delta_tiles(PassB a, TilePlan fwd, TilePlan rev) {
    extern __shared__ int4 s_pk[];  // the tile's records, its null records, its halo's; w: lambda x 2^18
    __shared__ float4 s_box[kTileBoxWords * kTileBoxes];
    __shared__ UpdateHead s_head;
    constexpr uint32_t B = T * L;
    float2 *s_kc = reinterpret_cast<float2 *>(s_pk + 2 * T + kTileHalo);  // their Gauss constants when widths differ
    const uint32_t n = a.d_len[kLenParticles];
    // the rows' form is the search's: it stays between the passes too
    const bool own = a.st->range_min == a.st->range_max || a.st->union_rows != 0u;
    const TilePlan &plan = own ? fwd : rev;
    const uint32_t *idx_arr = own ? a.idx : a.ridx;
    const uint32_t sub = threadIdx.x % L, rank = threadIdx.x / L;
    UpdateHead h;
    for (uint32_t tile = blockIdx.x; tile * T < n || tile == 0u; tile += gridDim.x) {
        const uint32_t base = tile * T;  // (as k_density_tiles starts)
        const uint4 head = plan.tile[tile];
        const uint32_t lane = plan.lane[base + rank];
        const uint2 *row = plan.rows + (size_t)tile * (T * kTileDepth / 4) + rank;
        const uint32_t *halo = plan.halo + (size_t)tile * kTileHalo;
        const uint32_t h0 = halo[threadIdx.x], h1 = halo[threadIdx.x + B];
        uint2 e = row[sub * T];
        if (tile == blockIdx.x) grid_dependency_trigger();
        const bool over = head.x == kHaloOver;
        const uint32_t H = over || n == 0u ? 0u : head.x;
        const bool valid = n != 0u && lane != kNoParticle;
        const uint32_t o = valid ? lane & 255u : 0u, j = base + o;
        const uint32_t cnt = valid ? lane >> 8 : 0u;
        const uint32_t depth = over ? 0u : min(cnt, (uint32_t)kTileDepth);
        const uint32_t corrections = own ? a.rcount[j] : 0u;
        if (threadIdx.x < min(a.nboxes, kTileBoxes)) tile_box(a, threadIdx.x, __uint_as_float(head.z), s_box);
        if (tile == blockIdx.x) {
            grid_dependency_wait();
            if (threadIdx.x < 32u) {  // its latency runs beside the staging's
                h = update_head<true>(a, n);
                if (threadIdx.x == 0) s_head = h;
            }
        }
        // everything the particle needs to its end, so that no load waits behind the row
        const int4 shj = valid ? a.shift[j] : make_int4(0, 0, 0, 0), fj = a.filt[j];
        const float2 kcj = a.kc[j];
        const int4 p = a.pk[j];  // w: the applied lambda
        const int pw = a.pos[j].w;  // the mass rides along
        const float pushed = a.prev_mode == 2 ? a.lam_prev[j] : 0.0f;
        const auto stage = [&](uint32_t k, uint32_t g) {
            int4 v = a.pk[g];
            v.w = __float_as_int(__int_as_float(v.w) * APBF_FIX);
            s_pk[k] = v;
            s_kc[k] = a.kc[g];
        };
        for (uint32_t k = threadIdx.x; k < T; k += B)
            if (n != 0u && k < head.y) {
                const int4 v = a.pk[base + k];
                s_pk[k] = make_int4(v.x, v.y, v.z, __float_as_int(__int_as_float(v.w) * APBF_FIX));
                s_pk[T + k] = make_int4(v.x, v.y, v.z, 0);
                s_kc[k] = s_kc[T + k] = a.kc[base + k];
            }
        if (threadIdx.x < H) stage(2 * T + threadIdx.x, h0);
        if (threadIdx.x + B < H) stage(2 * T + B + threadIdx.x, h1);
        for (uint32_t k = threadIdx.x + 2 * B; k < H; k += B) stage(2 * T + k, halo[k]);
        bool fil = false, hit = false, near = false;  // this particle's deferred filter, a neighbour cleared it or may have
        float3 ed = make_float3(0.f, 0.f, 0.f);
        if (shj.w != 0) fil = filter_dir(fj.x, fj.y, fj.z, ed);  // (only a deferred filter sets it)
        __syncthreads();
        if (tile == blockIdx.x) {
            h = s_head;
            if (h.skip) {
                update_skipped(a, h);
                return;
            }
            if (n == 0u) return;
            fil = fil && h.filter;
        }
        const GaussPair cj = gauss_pair(kcj.x, kcj.y);
        const int3 start = sub == 0 ? make_int3(shj.x, shj.y, shj.z) : make_int3(0, 0, 0);
        int3 acc = start;
        float low = 0.0f;
        {
            const F2 one = f2_pack(a.one, a.one);
            const F2 k36 = f2_pack(0.693147180559945309f * 0x1p19f, 0.693147180559945309f * 0x1p19f);
            const F2 ivd0 = f2_pack(cj.ivd36, cj.ivd36), norm0 = f2_pack(cj.norm, cj.norm), kk0 = f2_pack(cj.k2, cj.k2);
            const auto two = [&](uint32_t w, auto uniform, auto filter) {
                const uint32_t o0 = w & 0xffffu, o1 = w >> 16;
                const int4 q0 = tile_record(s_pk, o0), q1 = tile_record(s_pk, o1);
                const F2 dx = f2_pack((float)wadd(p.x, -q0.x), (float)wadd(p.x, -q1.x));
                const F2 dy = f2_pack((float)wadd(p.y, -q0.y), (float)wadd(p.y, -q1.y));
                const F2 dz = f2_pack((float)wadd(p.z, -q0.z), (float)wadd(p.z, -q1.z));
                const F2 r2 = dot3_f2(dx, dy, dz, dx, dy, dz, one);
                if (decltype(filter)::value) {
                    // gauss_filter_hit_fixed by squares, with margins a hundred times its
                    // rounding: above the upper line it hits, up to the lower it does not (nor
                    // below 0.0001 reference units, r2 < 688), between them the row is asked again
                    const F2 ex = f2_pack(ed.x, ed.x), ey = f2_pack(ed.y, ed.y), ez = f2_pack(ed.z, ed.z);
                    const float2 d = f2_unpack(dot3_f2(ex, ey, ez, dx, dy, dz, one));
                    const float2 lo = f2_unpack(r2 * f2_pack(0.35999f, 0.35999f));
                    const float2 hi = f2_unpack(f2_fma(r2, f2_pack(0.36001f, 0.36001f), f2_pack(700.0f, 700.0f)));
                    const float t0 = d.x * fabsf(d.x), t1 = d.y * fabsf(d.y);
                    near = near || t0 > lo.x || t1 > lo.y;
                    hit = hit || t0 > hi.x || t1 > hi.y;
                }
                F2 ivd = ivd0, norm = norm0, kk = kk0;
                if (!decltype(uniform)::value) {
                    const float2 c0 = *reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(s_kc) + o0 / 2u),
                                 c1 = *reinterpret_cast<const float2 *>(reinterpret_cast<const char *>(s_kc) + o1 / 2u);
                    ivd = f2_pack(c0.x, c1.x);
                    norm = f2_pack(c0.y, c1.y);
                    kk = ivd * k36;
                }
                F2 W, s;
                gauss_two(r2, ivd, norm, kk, low, W, s);
                const F2 sc = f2_pack(__int_as_float(q0.w), __int_as_float(q1.w));
                const float2 tx = f2_unpack((s * dx) * sc), ty = f2_unpack((s * dy) * sc), tz = f2_unpack((s * dz) * sc);
                acc.x = wadd(acc.x, wadd(f2i(tx.x), f2i(tx.y)));
                acc.y = wadd(acc.y, wadd(f2i(ty.x), f2i(ty.y)));
                acc.z = wadd(acc.z, wadd(f2i(tz.x), f2i(tz.y)));
            };
            const auto rows = [&](auto uniform, auto filter) {
                for (uint32_t k = sub * 4u; k < depth; k += L * 4u) {
                    const uint2 cur = e;
                    if (k + L * 4u < depth) e = row[(k / 4u + L) * T];
                    two(cur.x, uniform, filter);
                    if (k + 2u < depth) two(cur.y, uniform, filter);
                }
            };
            using Yes = std::true_type;
            using No = std::false_type;
            if (__any_sync(0xffffffffu, fil)) {  // one form per warp
                if (h.packed) rows(Yes(), Yes());
                else rows(No(), Yes());
                hit = hit && fil;
                if (fil && near && !hit) {
#pragma unroll 1
                    for (uint32_t k = 0; k < depth && !hit; ++k) {
                        const float3 D = udiff(tile_record(s_pk, row_offset(row[(k / 4u) * T], k)), p);
                        hit = gauss_filter_hit_fixed(ed, D, dot3x(D, D));
                    }
                }
            } else {
                if (h.packed) rows(Yes(), No());
                else rows(No(), No());
            }
        }
        const auto add = [&](int4 q, float sc, const GaussPair &gk, bool test) {
            const float3 D = udiff(q, p);
            const float r2 = dot3x(D, D);
            if (test && fil && !hit) hit = gauss_filter_hit_fixed(ed, D, r2);
            if (sc == 0.0f) return;
            float W;
            float3 g;
            gauss_terms_r2(D, r2, gk, W, g);
            acc.x = wadd(acc.x, f2i(g.x * sc));
            acc.y = wadd(acc.y, f2i(g.y * sc));
            acc.z = wadd(acc.z, f2i(g.z * sc));
        };
        if (L > 1) low = group_min<L>(low);  // the group sums its row again as one
        if (low < kLowExponent) {  // far out in a narrow kernel: subnormal results
            acc = start;
#pragma unroll 1
            for (uint32_t k = sub; k < depth; k += L) {
                const uint32_t of = row_offset(row[(k / 4u) * T], k);
                const int4 q = tile_record(s_pk, of);
                const float2 kk = h.packed ? kcj : s_kc[of / 16u];
                add(q, __int_as_float(q.w), gauss_pair(kk.x, kk.y), false);
            }
        }
        // what the tile does not hold, as in k_density_tiles
        const bool by_warp = head.w == 0u && cnt > kTileDepth;
        struct Gathered {
            int4 q;
            float2 k;
        };
        lane_row<L>(idx_arr + j, a.stride, depth + sub, by_warp ? (uint32_t)kTileDepth : cnt,
                    [&](uint32_t e) {
                        const uint32_t g = e & ~kNoDelta;
                        return Gathered{a.pk[g], h.packed ? kcj : a.kc[g]};
                    },
                    [&](const Gathered &x) {
                        add(x.q, __int_as_float(x.q.w) * APBF_FIX, gauss_pair(x.k.x, x.k.y), true);
                    });
        for (uint32_t left = __ballot_sync(0xffffffffu, sub == 0u && by_warp); left; left &= left - 1u) {
            const int src = __ffs(left) - 1;
            const WarpRow w(plan, idx_arr, a.stride, j, cnt, p, src);
            const float2 kw = make_float2(__shfl_sync(0xffffffffu, kcj.x, src), __shfl_sync(0xffffffffu, kcj.y, src));
            const bool test = __shfl_sync(0xffffffffu, fil && !hit ? 1 : 0, src) != 0;
            const float3 ew = make_float3(__shfl_sync(0xffffffffu, ed.x, src), __shfl_sync(0xffffffffu, ed.y, src),
                                          __shfl_sync(0xffffffffu, ed.z, src));
            int3 t = make_int3(0, 0, 0);
            bool any = false;
            w.each([&](uint32_t g) { return a.pk[g & ~kNoDelta]; }, [&](uint32_t g, const int4 &q) {
                const float3 D = udiff(q, w.p);
                const float r2 = dot3x(D, D);
                if (test && !any) any = gauss_filter_hit_fixed(ew, D, r2);
                const float lam = __int_as_float(q.w);
                if (lam == 0.0f) return;
                const float2 kk = h.packed ? kw : a.kc[g & ~kNoDelta];
                const int3 v = gauss_delta(D, r2, lam, gauss_pair(kk.x, kk.y));
                t.x = wadd(t.x, v.x);
                t.y = wadd(t.y, v.y);
                t.z = wadd(t.z, v.z);
            });
            t.x = __reduce_add_sync(0xffffffffu, t.x);
            t.y = __reduce_add_sync(0xffffffffu, t.y);
            t.z = __reduce_add_sync(0xffffffffu, t.z);
            any = __any_sync(0xffffffffu, any);
            if ((int)(threadIdx.x & 31u) == src) {
                acc.x = wadd(acc.x, t.x);
                acc.y = wadd(acc.y, t.y);
                acc.z = wadd(acc.z, t.z);
                hit = hit || any;
            }
        }
        if (h.corr) {  // the correction row (radii that differ): usually empty
            const uint32_t m = valid ? corrections : 0u;
            if (m)
                acc = h.packed ? delta_corrections<true, L, true>(a, a.pos, m, j, sub, p, cj, acc)
                               : delta_corrections<true, L, false>(a, a.pos, m, j, sub, p, cj, acc);
        }
        if (L > 1) {
            acc.x = group_wsum<L>(acc.x);
            acc.y = group_wsum<L>(acc.y);
            acc.z = group_wsum<L>(acc.z);
            if (h.filter) {
                int x = hit ? 1 : 0;
#pragma unroll
                for (int off = L / 2; off > 0; off >>= 1) x |= __shfl_xor_sync(0xffffffffu, x, off);
                hit = x != 0;
            }
        }
        if (valid && sub == 0) {
            const float lj = __int_as_float(p.w);
            uint32_t nb = h.nboxes, first = 0;
            int4 v = make_int4(wadd(p.x, acc.x), wadd(p.y, acc.y), wadd(p.z, acc.z), pw);
            if (nb && nb <= kTileBoxes) {
                first = tile_boxes_clear(v, s_box, nb);
                if (first == nb) {  // no box: box_push's round trip through FP32 and 2^-18
                    v.x = f2i((float)v.x);
                    v.y = f2i((float)v.y);
                    v.z = f2i((float)v.z);
                    nb = 0u;
                }
            }
            if (nb) v = box_push_from(v, a.radius[j], j, a.bmin, a.bmax, a.rot, first, nb);
            if (hit) a.bness[j] = 0.0f;
            a.pos_out[j] = v;
            if (a.prev_mode) a.lam_prev[j] = a.prev_mode == 1 ? lj : pushed + lj;
            accumulate(a.lam_acc, a.acc_mode, j, lj);
        }
        if (tile + gridDim.x < (n + T - 1) / T) __syncthreads();  // the shared records are the next tile's
    }
}

// ---- the solve loop as one persistent cooperative kernel ----

struct LoopArgs {
    int4 *pos_a;          // positions before the first loop pass; the final positions end here
    int4 *pos_b;          // the other position buffer
    uint32_t first;       // number of the first loop pass
    uint32_t max_passes;  // passes from this number on do not run
    uint32_t nboxes;      // boxes of the next iteration's collision (none after the last pass)
    int defer;            // the density pass may leave the Gauss filter to the position phase (rows symmetric)
};

constexpr uint32_t kBarrierSpins = 1u << 22;  // x __nanosleep(64): a few hundred ms at most

// Grid barrier of a cooperative launch (every block resident).  The last block to
// arrive finishes the density pass when fin is set (one thread, all partial sums
// in) and releases the others; a wait that exceeds kBarrierSpins sets
// APBF_FLAG_SPIN_LIMIT and returns false, after which the block leaves the kernel
// (the blocks still waiting give up in turn, so every wait ends).
__device__ __forceinline__ bool grid_barrier(Status *st, uint32_t &gen, const PassA *fin, uint32_t n) {
    __syncthreads();
    __shared__ uint32_t s_ok;
    if (threadIdx.x == 0) {
        uint32_t ok = 1u;
        __threadfence();
        const uint32_t arrived = atomicAdd(&st->bar_arrive, 1u) + 1u;
        if (arrived == gridDim.x) {
            if (fin) {
                const unsigned long long t1 = *(volatile unsigned long long *)&st->loop_e1;
                const unsigned long long t2 = *(volatile unsigned long long *)&st->loop_e2;
                st->loop_e1 = 0ull;
                st->loop_e2 = 0ull;
                finish_pass(fin->red_out, fin->st, fin->target, n, (long long)t1, (long long)t2,
                            error_meets_target(t1, n, fin->target, fin->target_m, fin->target_s));
            }
            st->bar_arrive = 0u;
            __threadfence();
            atomicAdd(&st->bar_gen, 1u);  // release
        } else {
            uint32_t spins = 0;
            bool inject;
            const uint32_t limit = wait_limit(st, kBarrierSpins, inject);
            while (inject || *(volatile uint32_t *)&st->bar_gen == gen) {
                if (++spins > limit) {
                    set_flag(st, APBF_FLAG_SPIN_LIMIT);
                    st->spin_where = 3u;
                    ok = 0u;
                    break;
                }
                __nanosleep(64);
            }
            __threadfence();
        }
        s_ok = ok;
    }
    __syncthreads();
    ++gen;
    return s_ok != 0u;
}

// Jacobi passes first .. max_passes-1 of a substep (or until a density pass meets
// the error target) in one launch: per pass, the density phase (density_one for
// every particle, error sums by integer atomics), a grid barrier whose last block
// finishes the pass, the position phase (delta_one) and a second barrier.  The
// per-particle arithmetic is the two-kernel form's own, so the results are
// identical; what goes away is two launches per pass and their ramp-up and drain.
// The widths' uniformity is the one pass 0 found (widths do not change within a
// substep).
template <bool GAUSS>
__global__ void __launch_bounds__(256, 4) k_solve_loop(PassA a, PassB b, LoopArgs l) {
    Status *st = a.st;
    if (a.early_exit && *(volatile uint32_t *)&st->converged) return;  // pass 0 met the target: no loop pass
    uint32_t gen = *(volatile uint32_t *)&st->bar_gen;  // read before this block's first arrival
    const uint32_t n = a.d_len[kLenParticles];
    const bool sym = st->range_min == st->range_max;
    const bool corr = !sym && st->union_rows != 0u;
    // with symmetric rows or correction rows the Gauss filter runs in the position phase
    // (as k_density_lambda decides)
    const bool defer = l.defer != 0 && (sym || corr);
    const bool packed = GAUSS && st->kw_uniform != 0u;
    const uint32_t *cnt_arr = sym || corr ? b.count : b.rcount;
    const uint32_t *idx_arr = sym || corr ? b.idx : b.ridx;
    const uint32_t T = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    int4 *cur = l.pos_a, *nxt = l.pos_b;
    for (uint32_t pass = l.first; pass < l.max_passes; ++pass) {
        PassSums ps;
        for (uint32_t i = t0; i < n; i += T) density_one<GAUSS, 1, false>(a, cur, i, n, 0u, defer, !GAUSS, ps);
        const PassSums bs = block_pass_sums(ps);
        if (threadIdx.x == 0) {
            atomicAdd(&st->loop_e1, (unsigned long long)bs.e1);
            atomicAdd(&st->loop_e2, (unsigned long long)bs.e2);
        }
        if (!grid_barrier(st, gen, &a, n)) return;
        if (*(volatile uint32_t *)&st->converged != 0u) {
            // converged: no position update (the positions stay in cur), the deferred
            // filter still belongs to this pass
            for (uint32_t j = t0; j < n; j += T) {
                if (defer) delta_skip_filter(b, cur, j);
                accumulate(b.lam_prev, b.prev_mode, j, 0.0f);
            }
            break;
        }
        const uint32_t nb = pass + 1u < l.max_passes ? l.nboxes : 0u;
        for (uint32_t j = t0; j < n; j += T)
            delta_one<GAUSS, 1>(b, cur, nxt, j, n, 0u, packed, defer, cnt_arr, idx_arr, corr, nb);
        if (!grid_barrier(st, gen, nullptr, n)) return;
        int4 *t = cur;
        cur = nxt;
        nxt = t;
    }
    if (cur != l.pos_a)  // an odd number of updates: bring the positions back to the caller's buffer
        for (uint32_t j = t0; j < n; j += T) l.pos_a[j] = cur[j];
}

// ---- the solve loops of a batch of scenes as one persistent cooperative kernel ----

// One scene of a batched solve: its pass arguments, its two position buffers and
// its loop limits (LoopArgs per scene).
struct BatchScene {
    PassA a;
    PassB b;
    LoopArgs l;
};

struct BatchSync {
    uint32_t bar_arrive;  // blocks arrived at the current grid barrier
    uint32_t bar_gen;     // grid barriers released so far
    uint32_t pad[2];
};

// Grid barrier of the batched solve (bounded like grid_barrier).  fin: the last
// block to arrive finishes the density pass of every scene that ran one (its
// threads one scene each: error means from the scenes' integer sums, convergence).
__device__ __forceinline__ bool batch_barrier(BatchSync *sy, uint32_t &gen, const BatchScene *tab, uint32_t S,
                                              unsigned long long *acc, const uint32_t *s_n, const uint8_t *s_run,
                                              bool fin) {
    __syncthreads();
    __shared__ uint32_t s_last, s_ok;
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&sy->bar_arrive, 1u) + 1u == gridDim.x ? 1u : 0u;
        s_ok = 1u;
    }
    __syncthreads();
    if (s_last) {
        __threadfence();
        if (fin)
            for (uint32_t sc = threadIdx.x; sc < S; sc += blockDim.x) {
                if (!s_run[sc]) continue;
                const unsigned long long t1 = *(volatile unsigned long long *)&acc[2 * sc];
                const unsigned long long t2 = *(volatile unsigned long long *)&acc[2 * sc + 1];
                acc[2 * sc] = 0ull;
                acc[2 * sc + 1] = 0ull;
                const PassA &pa = tab[sc].a;
                finish_pass(pa.red_out, pa.st, pa.target, s_n[sc], (long long)t1, (long long)t2,
                            error_meets_target(t1, s_n[sc], pa.target, pa.target_m, pa.target_s));
            }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            sy->bar_arrive = 0u;
            __threadfence();
            atomicAdd(&sy->bar_gen, 1u);  // release
        }
    } else if (threadIdx.x == 0) {
        uint32_t spins = 0;
        bool inject;
        const uint32_t limit = wait_limit(tab[0].a.st, kBarrierSpins, inject);
        while (inject || *(volatile uint32_t *)&sy->bar_gen == gen) {
            if (++spins > limit) {
                for (uint32_t sc = 0; sc < S; ++sc) {
                    set_flag(tab[sc].a.st, APBF_FLAG_SPIN_LIMIT);
                    tab[sc].a.st->spin_where = 4u;
                }
                s_ok = 0u;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
    }
    __syncthreads();
    ++gen;
    return s_ok != 0u;
}

constexpr uint32_t kBatchScenes = 256;  // scenes per batched solve (a finishing thread each)

// Jacobi passes 1.. of every scene in the table (each until its own error target or
// pass limit), the scenes' particles cut into units of one block: per pass the
// density phase of every running scene, a grid barrier whose last block finishes
// those scenes' passes, the position phase, a second barrier.  The per-particle
// arithmetic is density_one / delta_one, as in the per-scene forms, so each scene
// ends bit-identical to a solve of its own.
__global__ void __launch_bounds__(256, 4) k_solve_batch(const BatchScene *__restrict__ tab, uint32_t S,
                                                        BatchSync *sy, unsigned long long *acc) {
    __shared__ uint32_t s_n[kBatchScenes], s_unit[kBatchScenes + 1], s_max[kBatchScenes];
    __shared__ uint8_t s_run[kBatchScenes], s_conv[kBatchScenes], s_upd[kBatchScenes], s_done[kBatchScenes];
    __shared__ uint8_t s_defer[kBatchScenes], s_packed[kBatchScenes], s_sym[kBatchScenes];
    __shared__ uint32_t s_maxpass;
    uint32_t gen = *(volatile uint32_t *)&sy->bar_gen;  // read before this block's first arrival
    for (uint32_t sc = threadIdx.x; sc < S; sc += blockDim.x) {
        const BatchScene &b = tab[sc];
        const Status *st = b.a.st;
        s_n[sc] = b.a.d_len[kLenParticles];
        s_max[sc] = b.l.max_passes;
        // rows: 1 symmetric, 2 own rows with correction rows, 0 transposed
        s_sym[sc] = st->range_min == st->range_max ? 1 : (st->union_rows != 0u ? 2 : 0);
        s_defer[sc] = (b.l.defer != 0 && s_sym[sc] != 0) ? 1 : 0;
        s_packed[sc] = st->kw_uniform != 0u ? 1 : 0;
        s_done[sc] = (b.a.early_exit && *(volatile const uint32_t *)&st->converged) ? 1 : 0;  // pass 0 met the target
        s_upd[sc] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // units of blockDim particles per scene, and the largest pass limit
        uint32_t u = 0, mp = 0;
        for (uint32_t sc = 0; sc < S; ++sc) {
            s_unit[sc] = u;
            u += (s_n[sc] + blockDim.x - 1) / blockDim.x;
            mp = max(mp, s_max[sc]);
        }
        s_unit[S] = u;
        s_maxpass = mp;
    }
    __syncthreads();
    const uint32_t units = s_unit[S];
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t pass = 1; pass < s_maxpass; ++pass) {
        bool any = false;
        for (uint32_t sc = 0; sc < S; ++sc) any = any || (!s_done[sc] && pass < s_max[sc]);
        if (!any) break;  // uniform: every block holds the same flags
        __syncthreads();
        for (uint32_t sc = threadIdx.x; sc < S; sc += blockDim.x) s_run[sc] = (!s_done[sc] && pass < s_max[sc]) ? 1 : 0;
        __syncthreads();
        // density phase
        for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
            uint32_t lo = 0, hi = S;  // the scene of unit u: s_unit[sc] <= u < s_unit[sc + 1]
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_unit[mid] <= u) lo = mid;
                else hi = mid;
            }
            const uint32_t sc = lo;
            if (!s_run[sc]) continue;  // uniform over the block
            const BatchScene &bs = tab[sc];
            const int4 *cur = (s_upd[sc] & 1u) ? bs.l.pos_b : bs.l.pos_a;
            const uint32_t i = (u - s_unit[sc]) * blockDim.x + threadIdx.x;
            PassSums ps;
            density_one<true, 1, false>(bs.a, cur, i, s_n[sc], 0u, s_defer[sc] != 0, false, ps);
            long long e1 = ps.e1, e2 = ps.e2;
            for (int off = 16; off > 0; off >>= 1) {
                e1 += __shfl_down_sync(0xffffffffu, e1, off);
                e2 += __shfl_down_sync(0xffffffffu, e2, off);
            }
            if (lane == 0 && (e1 | e2)) {
                atomicAdd(&acc[2 * sc], (unsigned long long)e1);
                atomicAdd(&acc[2 * sc + 1], (unsigned long long)e2);
            }
        }
        if (!batch_barrier(sy, gen, tab, S, acc, s_n, s_run, true)) return;
        for (uint32_t sc = threadIdx.x; sc < S; sc += blockDim.x)
            s_conv[sc] = (s_run[sc] && *(volatile const uint32_t *)&tab[sc].a.st->converged) ? 1 : 0;
        __syncthreads();
        // position phase
        for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
            uint32_t lo = 0, hi = S;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_unit[mid] <= u) lo = mid;
                else hi = mid;
            }
            const uint32_t sc = lo;
            if (!s_run[sc]) continue;
            const BatchScene &bs = tab[sc];
            const PassB &b = bs.b;
            const int4 *cur = (s_upd[sc] & 1u) ? bs.l.pos_b : bs.l.pos_a;
            int4 *nxt = (s_upd[sc] & 1u) ? bs.l.pos_a : bs.l.pos_b;
            const uint32_t j = (u - s_unit[sc]) * blockDim.x + threadIdx.x;
            if (s_conv[sc]) {  // converged: the deferred filter of this pass, nothing applied
                if (j < s_n[sc]) {
                    if (s_defer[sc]) delta_skip_filter(b, cur, j);
                    accumulate(b.lam_prev, b.prev_mode, j, 0.0f);
                }
                continue;
            }
            const uint32_t nb = pass + 1u < s_max[sc] ? bs.l.nboxes : 0u;
            const uint32_t *cnt_arr = s_sym[sc] ? b.count : b.rcount;
            const uint32_t *idx_arr = s_sym[sc] ? b.idx : b.ridx;
            delta_one<true, 1>(b, cur, nxt, j, s_n[sc], 0u, s_packed[sc] != 0, s_defer[sc] != 0, cnt_arr, idx_arr,
                               s_sym[sc] == 2, nb);
        }
        if (!batch_barrier(sy, gen, tab, S, acc, s_n, s_run, false)) return;
        for (uint32_t sc = threadIdx.x; sc < S; sc += blockDim.x) {
            if (!s_run[sc]) continue;
            if (s_conv[sc]) s_done[sc] = 1;
            else s_upd[sc] = (uint8_t)(s_upd[sc] + 1);
        }
        __syncthreads();
    }
    // scenes that end after an odd number of updates: positions back to their pos_a
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        uint32_t lo = 0, hi = S;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s_unit[mid] <= u) lo = mid;
            else hi = mid;
        }
        const uint32_t sc = lo;
        if (!(s_upd[sc] & 1u)) continue;
        const uint32_t j = (u - s_unit[sc]) * blockDim.x + threadIdx.x;
        if (j < s_n[sc]) tab[sc].l.pos_a[j] = tab[sc].l.pos_b[j];
    }
}

__global__ void k_mass_volume(const float *inv_mass, const float *radius, const uint32_t *d_len, double *partials) {
    const uint32_t n = d_len[kLenParticles];
    double m = 0.0, v = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        m += 1.0 / (double)inv_mass[i];
        double r = radius[i];
        v += r * r * r;
    }
    __shared__ double s1[8], s2[8];
    for (int off = 16; off > 0; off >>= 1) {
        m += __shfl_down_sync(0xffffffffu, m, off);
        v += __shfl_down_sync(0xffffffffu, v, off);
    }
    if ((threadIdx.x & 31) == 0) {
        s1[threadIdx.x >> 5] = m;
        s2[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t1 = 0.0, t2 = 0.0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            t1 += s1[k];
            t2 += s2[k];
        }
        partials[2 * blockIdx.x] = t1;
        partials[2 * blockIdx.x + 1] = t2;
    }
}

__global__ void __launch_bounds__(256) k_finalize_mass(const double *partials, int blocks, double *out) {
    double t1, t2;
    block_sum2(partials, blocks, t1, t2);
    if (threadIdx.x == 0) {
        out[0] = t1;
        out[1] = t2;
    }
}

}  // namespace

// Calls f with std::integral_constant<int, L> for the tuned lanes per particle.
template <typename F>
void launch_lanes(int lanes, F &&f) {
    switch (lanes) {
        case 2: f(std::integral_constant<int, 2>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        default: f(std::integral_constant<int, 1>()); break;
    }
}

// Kernel arguments of the density pass (PassA) and the position update (PassB)
// for the context's current buffers and the solve options.
static PassA make_pass_a(apbf_ctx *ctx, const SolveOpts &o) {
    const bool converge = o.converge, projected = o.projected;
    const int feature_mode = o.feature_mode, prev_mode = o.prev_mode;
    FluidBufs &f = ctx->fl[ctx->fcur];
    const apbf_settings &st = ctx->settings;
    PassA a;
    a.pos = f.pos;
    a.inv_mass = f.inv_mass;
    a.radius = f.radius;
    a.kw = f.kernel_width;
    a.bness = f.boundariness;
    a.count = ctx->nb_count;
    a.idx = ctx->nb_idx;
    a.stride = ctx->row_stride;
    a.lambda = ctx->debug ? ctx->lambda : nullptr;
    a.shift = ctx->shift;
    a.rec = ctx->solve_rec;
    a.pk = ctx->solve_pk;
    a.kc = ctx->solve_kc;
    a.dbg_dens = ctx->debug ? ctx->dbg_density : nullptr;
    a.dbg_grad = ctx->dbg_grad;
    a.dbg_sq = ctx->dbg_sq;
    a.sync = ctx->pass_sync;
    a.d_len = ctx->d_len;
    a.st = ctx->status;
    a.red_out = ctx->red_out;
    a.target = converge ? st.density_error_target : 0.0f;
    split_target(a.target, a.target_m, a.target_s);
    a.early_exit = converge ? 1 : 0;
    a.features = feature_mode ? ctx->features : nullptr;
    a.selfdir = ctx->selfdir;
    a.vel = f.vel;
    a.lam_prev = f.lambda_prev;
    a.projected = projected && prev_mode == 2 ? 1 : 0;
    a.loop_offset = o.loop_offset;
    a.max_passes = o.max_passes;
    a.filt = ctx->tuning.filter_in_density ? nullptr : ctx->filt;
    const float rm2 = 2.0f * st.smallest_target_radius;
    a.rmin3 = rm2 * rm2 * rm2;
    a.one = 1.0f;
    a.hk = st.height_kernel_id;
    a.gk = st.gradient_kernel_id;
    a.method = st.boundariness_calculation_method;
    a.update_b = st.update_boundariness;
    a.b_speed = st.boundariness_adaption_speed;
    a.b_sgl_factor = st.boundariness_self_grad_length_factor;
    a.b_up_factor = st.boundariness_underpressure_factor;
    return a;
}

static PassB make_pass_b(apbf_ctx *ctx, const SolveOpts &o) {
    FluidBufs &f = ctx->fl[ctx->fcur];
    FluidBufs &alt = ctx->fl[ctx->fcur ^ 1];
    const apbf_settings &st = ctx->settings;
    PassB b;
    b.pos = f.pos;
    b.pos_out = alt.pos;
    b.rec = ctx->solve_rec;
    b.pk = ctx->solve_pk;
    b.kc = ctx->solve_kc;
    b.kw = f.kernel_width;
    b.shift = ctx->shift;
    b.radius = f.radius;
    b.bmin = ctx->box_min;
    b.bmax = ctx->box_max;
    b.rot = ctx->box_rot;
    b.nboxes = o.box_after ? ctx->n_boxes : 0u;
    b.count = ctx->nb_count;
    b.idx = ctx->nb_idx;
    b.rcount = ctx->rev_count;
    b.ridx = ctx->rev_idx;
    b.stride = ctx->row_stride;
    b.d_len = ctx->d_len;
    b.st = ctx->status;
    b.sync = ctx->pass_sync;
    b.red_out = ctx->red_out;
    b.target = o.converge ? st.density_error_target : 0.0f;
    split_target(b.target, b.target_m, b.target_s);
    b.one = 1.0f;
    b.gk = st.gradient_kernel_id;
    b.early_exit = o.converge ? 1 : 0;
    b.lam_prev = f.lambda_prev;
    b.lam_acc = ctx->lam_acc;
    b.prev_mode = o.prev_mode;
    b.acc_mode = o.acc_mode;
    b.loop_offset = o.loop_offset;
    b.max_passes = o.max_passes;
    b.loop_end = o.loop_end ? 1 : 0;
    b.loop_handle = o.loop_handle;
    b.filt = ctx->filt;
    b.bness = f.boundariness;
    return b;
}

// Launch shape of the two direct passes (launch_rules.cuh) and its grid.
static PassShape pass_shape(const apbf_ctx *ctx, bool features, int *grid) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    const apbf_tuning &t = ctx->tuning;
    const PassShape sh = pass_shape_rule({t.gather_lanes, t.pass_block, t.pass_blocks_per_sm}, cap, features);
    *grid = grid_for(ctx, (uint32_t)std::min<uint64_t>((uint64_t)cap * sh.lanes, 0xffffffffu), (int)sh.block,
                     (int)sh.per_sm);
    return sh;
}

// Calls f with the tile shape (particles, threads per particle) for the list.
template <typename F>
static void with_tile_shape(const apbf_ctx *ctx, F &&f) {
    if (tile_particles(ctx->cfg.particle_capacity) == 64u)
        f(std::integral_constant<int, 64>(), std::integral_constant<int, 2>());
    else
        f(std::integral_constant<int, 128>(), std::integral_constant<int, 1>());
}

// Rewriting the rows costs as much as about two passes gain by it, less where the passes
// are short of warps anyway: at 250 000 particles 40 us against 23 us a pass, at 2 197
// four passes are as fast with the direct kernels (273 against 285 us a frame).
bool tiles_wanted(const apbf_ctx *ctx) {
    const apbf_settings &st = ctx->settings;
    return st.height_kernel_id == 1 && st.gradient_kernel_id == 1 && st.boundariness_calculation_method != 1 &&
           st.solver_iterations >= (ctx->cfg.particle_capacity >= 65536u ? 4 : 6);
}

bool transposed_rows(const apbf_ctx *ctx) {
    const apbf_settings &st = ctx->settings;
    return ctx->search_method == APBF_NEIGHBORHOOD_BINARY_SEARCH ||
           (!st.basic_pbf && !st.base_kernel_width_on_boundary_distance);
}

bool tiles_eligible(const apbf_ctx *ctx) {
    return tiles_wanted(ctx) && ctx->tile_plan[0].halo && (!transposed_rows(ctx) || ctx->tile_plan[1].halo);
}

apbf_status tile_rows(apbf_ctx *ctx, cudaStream_t s) {
    const bool transposed = transposed_rows(ctx);
    apbf_status r = APBF_OK;
    with_tile_shape(ctx, [&](auto tc, auto) {
        constexpr int T = decltype(tc)::value;
        const uint32_t tiles = (ctx->cfg.particle_capacity + T - 1) / T;
        const int grid = (int)std::min<uint32_t>(std::max(tiles, 1u), (uint32_t)ctx->num_sms * 32u);
        for (int rev = 0; rev < (transposed ? 2 : 1) && r == APBF_OK; ++rev) {
            TileRowsArgs a;
            a.count = rev ? ctx->rev_count : ctx->nb_count;
            a.idx = rev ? ctx->rev_idx : ctx->nb_idx;
            a.stride = ctx->row_stride;
            a.d_len = ctx->d_len;
            a.st = ctx->status;
            a.reverse = rev;
            a.radius = ctx->fl[ctx->fcur].radius;
            a.plan = ctx->tile_plan[rev];
            r = [&]() -> apbf_status {
                APBF_BEFORE_LAUNCH(ctx, s, "k_tile_rows");
                k_tile_rows<T><<<grid, 256, 0, s>>>(a);
                APBF_AFTER_LAUNCH(ctx, s, "k_tile_rows");
                return APBF_OK;
            }();
        }
    });
    return r;
}

// One Jacobi pass over the tiles of the substep's rows.
// (The learned warm start's first pass gathers features and takes the direct kernels.)
static apbf_status launch_tiles(apbf_ctx *ctx, cudaStream_t s, const PassA &a, const PassB &b, const SolveOpts &o) {
    apbf_status r = APBF_OK;
    with_tile_shape(ctx, [&](auto tc, auto lc) {
        constexpr int T = decltype(tc)::value, L = decltype(lc)::value;
        const uint32_t tiles = (ctx->cfg.particle_capacity + T - 1) / T;
        const int grid = (int)std::min<uint32_t>(std::max(tiles, 1u), (uint32_t)ctx->num_sms * 64u);
        const size_t rec = (size_t)(2 * T + kTileHalo);
        r = [&]() -> apbf_status {
            APBF_BEFORE_LAUNCH(ctx, s, "k_density_tiles");
            // a pass behind a position update starts while that drains (the kernels wait for it
            // before they read what it wrote); the first kernel behind the rows does not, nor
            // do those of a batch, whose waiting blocks would keep other scenes' off the SMs
            // (16 scenes: 3113 against 3028 us)
            APBF_CUDA(launch_behind(o.later_pass && o.behind && !ctx->in_batch, k_density_tiles<T, L>, grid, T * L, rec * sizeof(int4), s, a,
                                    ctx->tile_plan[0]));
            APBF_AFTER_LAUNCH(ctx, s, "k_density_tiles");
            APBF_BEFORE_LAUNCH(ctx, s, "k_delta_tiles");
            APBF_CUDA(launch_behind(!ctx->in_batch, k_delta_tiles<T, L>, grid, T * L, rec * (sizeof(int4) + sizeof(float2)), s, b,
                                    ctx->tile_plan[0], ctx->tile_plan[1]));
            APBF_AFTER_LAUNCH(ctx, s, "k_delta_tiles");
            return APBF_OK;
        }();
    });
    return r;
}

apbf_status incompressibility(apbf_ctx *ctx, cudaStream_t s, const SolveOpts &o) {
    const bool learned = o.learned;
    FluidBufs &f = ctx->fl[ctx->fcur];
    FluidBufs &alt = ctx->fl[ctx->fcur ^ 1];
    const apbf_settings &st = ctx->settings;
    const bool gauss = st.height_kernel_id == 1 && st.gradient_kernel_id == 1;
    const PassA a = make_pass_a(ctx, o);
    int grid = 0;
    const PassShape sh = pass_shape(ctx, o.feature_mode != 0, &grid);
    const int lanes = (int)sh.lanes, pb = (int)sh.block;
    const bool xtra = a.features != nullptr || a.method == 1;
    if (o.tiles && gauss && !xtra) {
        const PassB b = make_pass_b(ctx, o);
        apbf_status r = launch_tiles(ctx, s, a, b, o);
        if (r != APBF_OK) return r;
        int4 *tmp = f.pos;
        f.pos = alt.pos;
        alt.pos = tmp;
        return APBF_OK;
    }
    // a pass starts behind a position update, the update behind its density pass: four passes
    // stage by stage over 19 683 particles 190 -> 180 us
    const bool first_behind = o.later_pass && o.behind && !ctx->in_batch;
    APBF_BEFORE_LAUNCH(ctx, s, "k_density_lambda");
    cudaError_t e = cudaSuccess;
    launch_lanes(lanes, [&](auto lc) {
        constexpr int Lc = decltype(lc)::value;
        if (gauss && xtra)
            e = launch_behind(first_behind, k_density_lambda<true, Lc, true>, grid, pb, 0, s, a);
        else if (gauss)
            e = launch_behind(first_behind, k_density_lambda<true, Lc, false>, grid, pb, 0, s, a);
        else
            e = launch_behind(first_behind, k_density_lambda<false, Lc, true>, grid, pb, 0, s, a);
    });
    APBF_CUDA(e);
    APBF_AFTER_LAUNCH(ctx, s, "k_density_lambda");

    if (learned) {  // the network's lambda replaces the plain one in this update
        apbf_status r = mlp_lambda(ctx, s, a.target, a.target_m, a.target_s);
        if (r != APBF_OK) return r;
    }
    const PassB b = make_pass_b(ctx, o);
    APBF_BEFORE_LAUNCH(ctx, s, "k_delta");
    launch_lanes(lanes, [&](auto lc) {
        constexpr int Lc = decltype(lc)::value;
        if (gauss)
            e = launch_behind(!learned && !ctx->in_batch, k_delta<true, Lc>, grid, pb, 0, s, b);
        else
            e = launch_behind(!learned && !ctx->in_batch, k_delta<false, Lc>, grid, pb, 0, s, b);
    });
    APBF_CUDA(e);
    APBF_AFTER_LAUNCH(ctx, s, "k_delta");
    // the updated positions now live in the alternate buffer: swap position buffers
    int4 *tmp = f.pos;
    f.pos = alt.pos;
    alt.pos = tmp;
    return APBF_OK;
}

// The tiled passes run behind one another with programmatic launches, so blocks of both
// kernels share an SM: they ask for the same split of its L1 (at different ones each
// launch waits for the SM to drain: 1760 against 1520 us for the 32 768-particle frame).
// 75 % shared memory holds every block the registers allow (50 %: 2213, 100 %: 2151
// against 2094 us at 119 771 particles).
apbf_status tiles_prepare_device() {
    constexpr int kShared = 75;
    constexpr auto kAttr = cudaFuncAttributePreferredSharedMemoryCarveout;
    APBF_CUDA(cudaFuncSetAttribute(k_density_tiles<64, 2>, kAttr, kShared));
    APBF_CUDA(cudaFuncSetAttribute(k_delta_tiles<64, 2>, kAttr, kShared));
    APBF_CUDA(cudaFuncSetAttribute(k_density_tiles<128, 1>, kAttr, kShared));
    APBF_CUDA(cudaFuncSetAttribute(k_delta_tiles<128, 1>, kAttr, kShared));
    return APBF_OK;
}

bool solve_persistent_eligible(const apbf_ctx *ctx, const SolveOpts &o) {
    const apbf_settings &st = ctx->settings;
    return ctx->persistent_solve && ctx->coop_blocks > 0 && !ctx->in_batch && st.height_kernel_id == 1 &&
           st.gradient_kernel_id == 1 &&
           st.boundariness_calculation_method != 1 && !o.feature_mode && !o.learned && !o.acc_mode &&
           !ctx->debug && !ctx->prof_on && o.max_passes >= 2;
}

apbf_status solve_persistent(apbf_ctx *ctx, cudaStream_t s, const SolveOpts &o) {
    if (!solve_persistent_eligible(ctx, o)) return APBF_ERR_INVALID_ARG;
    SolveOpts q = o;
    q.loop_offset = -1;
    q.box_after = true;  // decided per pass in the kernel
    PassA a = make_pass_a(ctx, q);
    PassB b = make_pass_b(ctx, q);
    a.features = nullptr;
    LoopArgs l;
    l.pos_a = ctx->fl[ctx->fcur].pos;
    l.pos_b = ctx->fl[ctx->fcur ^ 1].pos;
    l.first = 1u;
    l.max_passes = o.max_passes;
    l.nboxes = ctx->n_boxes;
    l.defer = (a.filt && a.method == 2) ? 1 : 0;
    // barrier counters and pass sums start from zero on every launch
    APBF_CUDA(cudaMemsetAsync(&ctx->status->bar_arrive, 0,
                              offsetof(Status, loop_e2) + sizeof(unsigned long long) - offsetof(Status, bar_arrive), s));
    const uint32_t want = (ctx->cfg.particle_capacity + 255u) / 256u;
    const uint32_t grid = std::max(1u, std::min((uint32_t)ctx->coop_blocks, want));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    APBF_BEFORE_LAUNCH(ctx, s, "k_solve_loop");
    APBF_CUDA(cudaLaunchKernelEx(&cfg, k_solve_loop<true>, a, b, l));
    APBF_AFTER_LAUNCH(ctx, s, "k_solve_loop");
    return APBF_OK;
}

// Resident blocks of the persistent solve kernel (0: cooperative launches are
// not available), computed once per context.
int solve_persistent_blocks(int device, int num_sms) {
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_loop<true>, 256, 0) != cudaSuccess) return 0;
    return per_sm * num_sms;
}

bool batch_solve_eligible(const apbf_ctx *ctx, const SolveOpts &o) {
    const apbf_settings &st = ctx->settings;
    return ctx->coop_blocks > 0 && st.height_kernel_id == 1 && st.gradient_kernel_id == 1 &&
           st.boundariness_calculation_method != 1 && !o.feature_mode && !o.learned && !o.acc_mode && !ctx->debug &&
           !ctx->prof_on && o.max_passes >= 2;
}

size_t batch_scene_bytes() { return sizeof(BatchScene); }
size_t batch_sync_bytes() { return sizeof(BatchSync); }
uint32_t batch_max_scenes() { return kBatchScenes; }

void batch_scene_fill(apbf_ctx *ctx, const SolveOpts &o, void *entry) {
    SolveOpts q = o;
    q.loop_offset = -1;
    q.box_after = true;  // decided per pass in the kernel
    BatchScene &e = *reinterpret_cast<BatchScene *>(entry);
    e.a = make_pass_a(ctx, q);
    e.a.features = nullptr;
    e.b = make_pass_b(ctx, q);
    e.l.pos_a = ctx->fl[ctx->fcur].pos;
    e.l.pos_b = ctx->fl[ctx->fcur ^ 1].pos;
    e.l.first = 1u;
    e.l.max_passes = o.max_passes;
    e.l.nboxes = ctx->n_boxes;
    e.l.defer = (e.a.filt && e.a.method == 2) ? 1 : 0;
}

apbf_status solve_batch_launch(const void *d_table, uint32_t n_scenes, void *d_sync, unsigned long long *d_acc,
                               int grid, cudaStream_t s) {
    if (n_scenes == 0 || n_scenes > kBatchScenes || grid <= 0) return APBF_ERR_INVALID_ARG;
    APBF_CUDA(cudaMemsetAsync(d_sync, 0, sizeof(BatchSync), s));
    APBF_CUDA(cudaMemsetAsync(d_acc, 0, (size_t)2 * n_scenes * sizeof(unsigned long long), s));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    APBF_CUDA(cudaLaunchKernelEx(&cfg, k_solve_batch, reinterpret_cast<const BatchScene *>(d_table), n_scenes,
                                 reinterpret_cast<BatchSync *>(d_sync), d_acc));
    return APBF_OK;
}

int solve_batch_blocks(int device, int num_sms) {
    int coop = 0;
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_batch, 256, 0) != cudaSuccess) return 0;
    return per_sm * num_sms;
}

apbf_status reduce_fp64(apbf_ctx *ctx, double out[4], cudaStream_t s) {
    FluidBufs &f = ctx->fl[ctx->fcur];
    const int g = ctx->red_blocks;
    // red_out[2..3] hold the error of the last density pass (the position update behind it wrote them)
    APBF_BEFORE_LAUNCH(ctx, s, "k_mass_volume");
    k_mass_volume<<<g, kBlock, 0, s>>>(f.inv_mass, f.radius, ctx->d_len, ctx->red_partials + 4 * g);
    APBF_AFTER_LAUNCH(ctx, s, "k_mass_volume");
    APBF_BEFORE_LAUNCH(ctx, s, "k_finalize_mass");
    k_finalize_mass<<<1, 256, 0, s>>>(ctx->red_partials + 4 * g, g, ctx->red_out);
    APBF_AFTER_LAUNCH(ctx, s, "k_finalize_mass");
    APBF_CUDA(cudaMemcpyAsync(out, ctx->red_out, 4 * sizeof(double), cudaMemcpyDeviceToHost, s));
    APBF_CUDA(cudaStreamSynchronize(s));
    return APBF_OK;
}

namespace {
// Appends (features, sum of min(0, lambda)) of the particles to the caller's
// sample buffers, in particle order, up to their capacity.
__global__ void k_record_append(const float *feat, const float *acc, const uint32_t *d_len, float *out_f,
                                float *out_t, uint32_t cap, uint32_t *count) {
    const uint32_t n = d_len[kLenParticles];
    const uint32_t base = *count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t r = base + i;
        if (r >= cap) break;
        for (int k = 0; k < 8; ++k) out_f[(size_t)r * 8 + k] = feat[(size_t)i * 8 + k];
        out_t[r] = acc[i];
    }
}
__global__ void k_record_count(const uint32_t *d_len, uint32_t cap, uint32_t *count) {
    const uint32_t v = *count + d_len[kLenParticles];
    *count = v < cap ? v : cap;
}
}  // namespace

apbf_status record_samples(apbf_ctx *ctx, cudaStream_t s) {
    const uint32_t cap = ctx->cfg.particle_capacity;
    APBF_BEFORE_LAUNCH(ctx, s, "k_record_append");
    k_record_append<<<grid_for(ctx, cap), kBlock, 0, s>>>(ctx->features, ctx->lam_acc, ctx->d_len, ctx->rec_features,
                                                         ctx->rec_targets, ctx->rec_capacity, ctx->rec_count);
    APBF_AFTER_LAUNCH(ctx, s, "k_record_append");
    APBF_BEFORE_LAUNCH(ctx, s, "k_record_count");
    k_record_count<<<1, 1, 0, s>>>(ctx->d_len, ctx->rec_capacity, ctx->rec_count);
    APBF_AFTER_LAUNCH(ctx, s, "k_record_count");
    return APBF_OK;
}

}  // namespace apbf
