// mc_march.cuh -- the device helpers of the marches (Philox, Sobol', the
// attenuation and trigonometric polynomials, table lookups, the control
// variate's straight flight, the ray's direction, slab and tally) and the
// launch helpers; the fine-grid two-cell marches are in mc_march_pair.cuh, the
// multigrid march in mc_march_mg.cuh.  The march translation units are compiled with
// -fmad=false: the arithmetic is written with explicit fmaf so the host
// replay (oracle/mc_oracle.cpp) reproduces every ray bit for bit; exp, log,
// sin and cos are the project's own polynomial kernels for the same reason.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "mc_internal.h"
#include "../../include/dnsmc.h"

namespace dnsmc {

// ---------------------------------------------------------------------------
// Philox4x32-10 counter-based generator (Salmon, Moraes, Dror, Shaw,
// "Parallel random numbers: as easy as 1, 2, 3", SC'11).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r > 0) { k0 += 0x9E3779B9u; k1 += 0xBB67AE85u; }
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
    }
    return c;
}

// ---------------------------------------------------------------------------
// expm1 for x <= 0: Cody-Waite reduction x = n*ln2 + r, then expm1(r) =
// r (1 + r g(r)) with g(r) = (e^r - 1 - r)/r^2 replaced by its degree-4
// minimax polynomial on [-ln2/2, ln2/2] (Remez exchange computed for this
// project; |error| 6.2e-8 on g), then 2^n expm1(r) + (2^n - 1).  n is
// rounded by the shifter sh = fmaf(x, log2(e), 1.5 * 2^23): the sum lies in
// [2^23, 2^24), where the float spacing is 1, so sh - 1.5 * 2^23 is an
// integer within 1/2 (plus the fma's rounding) of x log2(e), and the low bits
// of sh hold n itself, so 2^n is one integer multiply-add on them.  Only +,
// *, fmaf and integer bit operations: bit-identical on any IEEE-754 machine.
// ---------------------------------------------------------------------------
constexpr float kExpShift = 12582912.0f;           // 1.5 * 2^23, bits 0x4B400000
__device__ __forceinline__ float mc_pow2_from_shift(float sh) {
    // bits(sh) = 0x4B400000 + n, so (n + 127) << 23 is bits(sh) << 23 plus a
    // constant, modulo 2^32
    return __uint_as_float((__float_as_uint(sh) << 23) + ((127u - 0x4B400000u) << 23));
}
__device__ __forceinline__ float mc_expm1(float x) {
    x = fmaxf(x, -87.0f);                          // n in [-126, 0]
    const float sh = fmaf(x, 1.44269504088896341f, kExpShift);
    const float n = sh - kExpShift;
    float r = fmaf(n, -0.693145751953125f, x);
    r = fmaf(n, -1.42860682030941723212e-6f, r);
    float q = 1.39411131385713816e-3f;
    q = fmaf(q, r, 8.36317520588636398e-3f);
    q = fmaf(q, r, 4.16663736104965210e-2f);
    q = fmaf(q, r, 1.66665762662887573e-1f);
    q = fmaf(q, r, 0.5f);
    float p = fmaf(q, r, 1.0f);
    p = p * r;                                     // expm1(r)
    const float two_n = mc_pow2_from_shift(sh);
    return fmaf(two_n, p, two_n - 1.0f);
}

// mc_expm1 of two arguments at once with paired FP32 instructions
// (f32x2 add / mul / fma, each half rounded to nearest like its scalar
// form): the same operations in the same order, so each half is
// bit-identical to mc_expm1 of it.  Used for the two cells of a lane.
__device__ __forceinline__ float2 mc_expm1_x2(float2 x) {
    x.x = fmaxf(x.x, -87.0f);
    x.y = fmaxf(x.y, -87.0f);
    const float2 sh = __ffma2_rn(x, make_float2(1.44269504088896341f, 1.44269504088896341f),
                                 make_float2(kExpShift, kExpShift));
    const float2 n = __fadd2_rn(sh, make_float2(-kExpShift, -kExpShift));
    float2 r = __ffma2_rn(n, make_float2(-0.693145751953125f, -0.693145751953125f), x);
    r = __ffma2_rn(n, make_float2(-1.42860682030941723212e-6f, -1.42860682030941723212e-6f), r);
    float2 q = __ffma2_rn(make_float2(1.39411131385713816e-3f, 1.39411131385713816e-3f), r,
                          make_float2(8.36317520588636398e-3f, 8.36317520588636398e-3f));
    q = __ffma2_rn(q, r, make_float2(4.16663736104965210e-2f, 4.16663736104965210e-2f));
    q = __ffma2_rn(q, r, make_float2(1.66665762662887573e-1f, 1.66665762662887573e-1f));
    q = __ffma2_rn(q, r, make_float2(0.5f, 0.5f));
    float2 p = __ffma2_rn(q, r, make_float2(1.0f, 1.0f));
    p = __fmul2_rn(p, r);
    const float2 two_n = make_float2(mc_pow2_from_shift(sh.x), mc_pow2_from_shift(sh.y));
    return __ffma2_rn(two_n, p, __fadd2_rn(two_n, make_float2(-1.0f, -1.0f)));
}

// sin and cos of x in [0, pi/4]: Taylor series to x^11 / x^12.
__device__ __forceinline__ void mc_sincos_oct(float x, float *s, float *c) {
    const float z = x * x;
    float ps = -2.50521083854417188e-8f;           // -1/11!
    ps = fmaf(ps, z, 2.75573192239858907e-6f);     //  1/9!
    ps = fmaf(ps, z, -1.98412698412698413e-4f);    // -1/7!
    ps = fmaf(ps, z, 8.33333333333333333e-3f);     //  1/5!
    ps = fmaf(ps, z, -1.66666666666666667e-1f);    // -1/3!
    *s = fmaf(ps * z, x, x);
    float pc = 2.08767569878680990e-9f;            //  1/12!
    pc = fmaf(pc, z, -2.75573192239858907e-7f);    // -1/10!
    pc = fmaf(pc, z, 2.48015873015873016e-5f);     //  1/8!
    pc = fmaf(pc, z, -1.38888888888888889e-3f);    // -1/6!
    pc = fmaf(pc, z, 4.16666666666666667e-2f);     //  1/4!
    pc = fmaf(pc, z, -0.5f);
    *c = fmaf(pc, z, 1.0f);
}

// cos and sin of 2*pi*m/2^24 for a 24-bit integer m: exact quadrant and
// octant reduction on the integer, polynomial on [0, pi/4].
__device__ __forceinline__ void mc_sincos_turn(uint32_t m, float *cs, float *sn) {
    const uint32_t q = m >> 22;
    const uint32_t r = m & 0x3FFFFFu;
    const bool hi = r > 0x200000u;
    const float th = (float)(hi ? (0x400000u - r) : r) * 3.74507028e-7f;  // pi*2^-23
    float s, c;
    mc_sincos_oct(th, &s, &c);
    const float cq = hi ? s : c, sq = hi ? c : s;
    float co, si;
    switch (q) {
        case 0: co = cq;  si = sq;  break;
        case 1: co = -sq; si = cq;  break;
        case 2: co = -cq; si = -sq; break;
        default: co = sq; si = -cq; break;
    }
    *cs = co; *sn = si;
}

// Sobol' direction numbers of the four sampled dimensions (host-computed).
static __constant__ uint32_t c_sobol[4][32];  // one copy per translation unit

__device__ __forceinline__ uint4 sobol4(uint32_t m) {
    uint32_t a = 0, b = 0, c = 0, d = 0;
    while (m) {  // one pass per set bit of m
        const int k = __ffs(m) - 1;
        a ^= c_sobol[0][k]; b ^= c_sobol[1][k]; c ^= c_sobol[2][k]; d ^= c_sobol[3][k];
        m &= m - 1u;
    }
    return make_uint4(a, b, c, d);
}

__device__ __forceinline__ float u24(uint32_t x) { return (float)(x >> 8) * 5.9604644775390625e-8f; }

// Linear position in a uniform grid of n points, clamped as the reference's
// clamp-addressed linear-filter textures (code/memory_copy.cu:245-247).
__device__ __forceinline__ void grid_pos(float v, float v0, float inv, int n, int *i, float *f) {
    float p = (v - v0) * inv;
    p = fminf(fmaxf(p, 0.0f), (float)(n - 1));
    int ii = (int)p;
    ii = min(ii, n - 2);
    *i = ii;
    *f = p - (float)ii;
}

// Split a clamped table coordinate p in [0, n-1] into cell and fraction.
__device__ __forceinline__ void pos_split(float p, int n, int *i, float *f) {
    int ii = (int)p;
    ii = min(ii, n - 2);
    *i = ii;
    *f = p - (float)ii;
}

// Paired tables: the k part of a sample's slab holds, per table cell
// kidx = ti*(nX-1) + xi of an x-table, the 16-byte entry (k[t][x],
// k[t][x+1] - k[t][x], k[t+1][x], k[t+1][x+1] - k[t+1][x]) for t = ti <=
// nT - 2, or per ti the pair (k[t], k[t+1] - k[t]); its Ib part holds (Ib[t],
// Ib[t+1] - Ib[t]) of the sample's band.  A bilinear lookup is one 16-byte
// load and three fmaf (the differences are the same FP32 subtractions the
// interpolation would do).  The march reads them from the warp's copy of the
// slab in shared memory.
template <int MODE>
__device__ __forceinline__ float lookup_k(const float2 *ks, int kidx, float ft, float fx) {
    if (MODE == MODE_TX) {
        const float4 v = reinterpret_cast<const float4 *>(ks)[kidx];
        const float2 a = make_float2(v.x, v.y), b = make_float2(v.z, v.w);
        const float k0 = fmaf(fx, a.y, a.x);
        const float k1 = fmaf(fx, b.y, b.x);
        return fmaf(ft, k1 - k0, k0);
    } else {
        const float2 a = ks[kidx];
        return fmaf(ft, a.y, a.x);
    }
}

__device__ __forceinline__ float lookup_ib(const float2 *ibs, int ti, float ft) {
    const float2 a = ibs[ti];
    return fmaf(ft, a.y, a.x);
}

// Field element type of the march: T (grey), or the cell's table coordinates.
template <int MODE> struct FieldT { typedef float type; };
template <> struct FieldT<MODE_T> { typedef int2 type; };
template <> struct FieldT<MODE_TX> { typedef int4 type; };

// (k index, T cell, T fraction, x fraction) of a table-coordinate element
template <int MODE>
__device__ __forceinline__ void cell_coords(const typename FieldT<MODE>::type &v, int *kidx, int *ti, float *ft,
                                            float *fx) {
    if constexpr (MODE == MODE_TX) {
        *kidx = v.x; *ft = __int_as_float(v.y); *fx = __int_as_float(v.z); *ti = v.w;
    } else if constexpr (MODE == MODE_T) {
        *kidx = v.x; *ti = v.x; *ft = __int_as_float(v.y); *fx = 0.0f;
    }
}

// ---------------------------------------------------------------------------
// -ln(u) for u in (0, 1): u = m 2^e with m in [sqrt(1/2), sqrt(2)),
// ln m = 2 atanh(s), s = (m - 1)/(m + 1), odd series to s^11 (|s| <= 0.1716,
// truncation below 1e-9); e ln 2 split Cody-Waite.  +, *, /, fmaf only.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float mc_neglog(float u) {
    uint32_t b = __float_as_uint(u);
    int e = (int)((b >> 23) & 0xffu) - 127;
    float m = __uint_as_float((b & 0x7fffffu) | 0x3f800000u);
    if (m > 1.41421356f) { m = m * 0.5f; e += 1; }
    const float s = (m - 1.0f) / (m + 1.0f);
    const float z = s * s;
    float p = 9.09090909090909091e-2f;            // 1/11
    p = fmaf(p, z, 1.11111111111111111e-1f);       // 1/9
    p = fmaf(p, z, 1.42857142857142857e-1f);       // 1/7
    p = fmaf(p, z, 2.0e-1f);                       // 1/5
    p = fmaf(p, z, 3.33333333333333333e-1f);       // 1/3
    p = fmaf(p, z, 1.0f);
    const float lnm = 2.0f * s * p;
    const float fe = (float)e;
    const float ln = fmaf(fe, 0.693145751953125f, fmaf(fe, 1.42860682030941723212e-6f, lnm));
    return -ln;
}

// uniform in (0, 1) from the top 24 bits
__device__ __forceinline__ float u24o(uint32_t x) { return ((float)(x >> 8) + 0.5f) * 5.9604644775390625e-8f; }

// Henyey-Greenstein scattering (asymmetry g): the cosine and sine of the angle
// from a uniform word, and the new direction from them and the azimuth's.
__device__ __forceinline__ void hg_angle(float g, uint32_t uc, float *cos_t, float *sin_t) {
    const float u = u24(uc);
    float ct;
    if (fabsf(g) < 1e-6f) {
        ct = 1.0f - 2.0f * u;
    } else {
        const float tmp = (1.0f - g * g) / (1.0f - g + 2.0f * g * u);
        ct = (1.0f + g * g - tmp * tmp) / (2.0f * g);
    }
    ct = fminf(fmaxf(ct, -1.0f), 1.0f);
    *cos_t = ct;
    *sin_t = sqrtf(fmaxf(0.0f, 1.0f - ct * ct));
}
__device__ __forceinline__ void hg_turn(float ct, float st, float cph, float sph, float *sW, float *sA, float *sB) {
    const float w = *sW, a = *sA, b = *sB;
    float nw, na, nb;
    if (fabsf(w) > 0.99999f) {
        na = st * cph;
        nb = st * sph;
        nw = w > 0.0f ? ct : -ct;
    } else {
        const float tmp = sqrtf(1.0f - w * w);
        na = st * (a * w * cph - b * sph) / tmp + a * ct;
        nb = st * (b * w * cph + a * sph) / tmp + b * ct;
        nw = -st * cph * tmp + w * ct;
    }
    *sW = nw; *sA = na; *sB = nb;
}

// Surrogate of the control variate: the ray's straight flight through the
// layer-mean medium, read from its table row (the ray's field, spectral
// sample and layer; cv_table_kernel) by linear interpolation in
// u = sqrt(|sW|) between the nodes m / kSurBins.  Returns the collected
// intensity J and the own-layer absorptance A.  The reads are warp-uniform.
__device__ __forceinline__ void surrogate_lookup(const float4 *row, float sW, float *J, float *A) {
    const float x = sqrtf(fabsf(sW)) * (float)kSurBins;
    const int m = min((int)x, kSurBins - 1);
    const float r = x - (float)m;
    const float4 e = __ldg(row + (sW > 0.0f ? kSurBins : 0) + m);
    *J = fmaf(r, e.y, e.x);
    *A = fmaf(r, e.w, e.z);
}

// ---------------------------------------------------------------------------
// Pieces shared by the marches: a packet-ray's direction, the copy of its spectral sample's table slab, one ray's tally.
// ---------------------------------------------------------------------------

// Isotropic direction (the reference's emiss_ang, code/mc_gpu.cu:813-820):
// cos(theta) = 1 - 2u from the top 24 bits of x.y, phi = 2 pi u' from x.x.
__device__ __forceinline__ void ray_direction(uint4 x, float *sW, float *sA, float *sB) {
    const float mu = fmaf((float)(x.y >> 8), -1.1920928955078125e-7f, 1.0f);
    const float st = sqrtf(fmaxf(0.0f, fmaf(-mu, mu, 1.0f)));
    float cph, sph;
    mc_sincos_turn(x.x >> 8, &cph, &sph);
    *sW = mu;
    *sA = st * cph;
    *sB = st * sph;
}

// ---------------------------------------------------------------------------
// The ray's table slab arrives by one bulk copy of the TMA engine
// (cp.async.bulk, global -> this CTA's shared memory) that signals the warp's
// transaction barrier (mbarrier) in shared memory; the warp waits on the
// barrier's phase parity.  Each warp owns one barrier and one slab buffer.
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Lane 0 initialises the warp's barrier (one arrival per phase: the issuing
// lane's arrive.expect_tx) before the warp's first copy.
__device__ __forceinline__ void slab_bar_init(uint64_t *bar, int lane) {
    if (lane == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
}

// Bounded wait (at most `polls` polls) for the barrier phase of the given
// parity to complete.
__device__ __forceinline__ bool slab_bar_wait(const uint64_t *bar, uint32_t parity, int polls) {
    const uint32_t b = smem_addr(bar);
    for (int it = 0; it < polls; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(b), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// The sample's slab (k, then Ib of its band; slab_len * 8 bytes, a multiple
// of 16 at a 16-byte aligned address on both sides) into this warp's shared
// copy: slab_issue starts the copy once the previous ray's lookups are done
// (the warp converges, and the async proxy is ordered after the generic
// one), slab_wait waits for it.  *phase is the warp's
// barrier parity, flipped per completed copy.  The first wait polls
// P.slab_polls0 times (kSlabWaitPolls; fewer only in tests of this path).
// A wait that runs out sets DNSMC_STATUS_COPY_TIMEOUT (the host reports the
// solve as failed) and waits once more; if the copy has still not arrived,
// returns false with the phase unchanged: the warp then takes no further
// copies or items and calls slab_drain before it exits.  The outcome is
// the same in every lane of the warp.
__device__ __forceinline__ void slab_issue(const MarchParams &P, int sid, uint32_t slab, int lane, uint64_t *bar) {
    __syncwarp();
    if (lane == 0) {
        const uint32_t bytes = (uint32_t)P.slab_len * 8u;
        const float2 *src = P.slab + (long long)sid * P.slab_len;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                     : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         slab),
                     "l"(src), "r"(bytes), "r"(smem_addr(bar))
                     : "memory");
    }
}

__device__ __forceinline__ bool slab_wait(const MarchParams &P, uint64_t *bar, uint32_t *phase, unsigned int *flags) {
    if (!__all_sync(0xffffffffu, slab_bar_wait(bar, *phase, P.slab_polls0))) {
        *flags |= DNSMC_STATUS_COPY_TIMEOUT;
        if (!__all_sync(0xffffffffu, slab_bar_wait(bar, *phase, kSlabWaitPolls))) return false;
    }
    *phase ^= 1u;
    return true;
}

// Before a warp whose copy did not arrive exits: one more bounded wait for
// that copy, so that it does not land in shared memory the next block on
// this SM may own.
__device__ __forceinline__ void slab_drain(const uint64_t *bar, uint32_t phase) {
    slab_bar_wait(bar, phase, kSlabWaitPolls);
}

// Float pairs (hi, lo): about 48 bits at FP32 rates (error-free sums; the
// translation units of the marches are compiled without FMA contraction, so
// the error terms stay exact).  This GPU's FP64 rate is a small fraction of
// its FP32 rate, and a warp's FP64 instructions at the end of every ray
// held the march up.
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
    const float s = a.x + b.x;
    const float bb = s - a.x;
    float e = (a.x - (s - bb)) + (b.x - bb);
    e = e + (a.y + b.y);
    const float hi = s + e;
    return make_float2(hi, e - (hi - s));
}
__device__ __forceinline__ float2 ff_addf(float2 a, float b) {
    const float s = a.x + b;
    const float bb = s - a.x;
    float e = (a.x - (s - bb)) + (b - bb);
    e = e + a.y;
    const float hi = s + e;
    return make_float2(hi, e - (hi - s));
}
__device__ __forceinline__ double ff_value(float2 a) { return (double)a.x + (double)a.y; }

// One ray of a cell into its sums, as float pairs: the sum, and the sum of
// squares (iid) or of the squared replicate means (RQMC: *rep holds the
// running replicate sum, m the ray's index in its replicate of M rays; the
// mean is the pair divided by M, its remainder exact by fma).
__device__ __forceinline__ void tally_ray(const MarchParams &P, float X, int m, int M, float2 *sum, float2 *sq,
                                          float2 *rep) {
    *sum = ff_addf(*sum, X);
    if (P.sampler) {
        const float2 Sb = ff_addf(*rep, X);
        if (m == M - 1) {  // end of a replicate: accumulate its mean squared
            const float Mf = (float)M;
            const float q = Sb.x / Mf;
            const float ql = (fmaf(-q, Mf, Sb.x) + Sb.y) / Mf;
            const float p = q * q;
            *sq = ff_add(*sq, make_float2(p, fmaf(q, q, -p) + 2.0f * (q * ql)));
            *rep = make_float2(0.0f, 0.0f);
        } else {
            *rep = Sb;
        }
    } else {
        const float p = X * X;
        *sq = ff_add(*sq, make_float2(p, fmaf(X, X, -p)));
    }
}

// Rays [rbeg, rend) of a unit: part `part` of an item of N rays.
__device__ __forceinline__ void unit_rays(const MarchParams &P, int part, int N, int *rbeg, int *rend) {
    const int per = (N + P.parts - 1) / P.parts;
    *rbeg = min(part * per, N);
    *rend = min(*rbeg + per, N);
}

// A warp has stored a unit's contributions (rayx): whether it was the item's
// last unit.  The result is the same in every lane.
__device__ __forceinline__ bool unit_done(const MarchParams &P, long long item, int lane) {
    __threadfence();
    __syncwarp();
    unsigned int n = 0;
    if (lane == 0) n = atomicAdd(P.parts_done + item, 1u);
    n = __shfl_sync(0xffffffffu, n, 0);
    __threadfence();
    return n == (unsigned int)P.parts - 1u;
}

// Sums of one cell of an item over its N rays in ray order (x: the cell's
// first contribution, CELLS values a ray), as tally_ray adds them.  Eight rays'
// values are fetched together; the multigrid march (CELLS = 32), whose steps
// fill the instruction cache, takes a loop of one ray with four fetched ahead
// (64^3, five levels: 1.41 -> 1.37 ms; the fine marches lose by it: grey 64^3
// 2.91 -> 2.98 ms).
template <int CELLS>
__device__ __forceinline__ double2 sum_rays(const MarchParams &P, const float *x, int N, int M) {
    float2 sum = make_float2(0.0f, 0.0f), sq = sum, rep = sum;
    int m = 0;
    if constexpr (CELLS == 32) {
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = q < N ? __ldcg(x + (long long)q * CELLS) : 0.0f;
#pragma unroll 1
        for (int r = 0; r < N; ++r) {
            tally_ray(P, v[0], m, M, &sum, &sq, &rep);
            m = P.sampler && m == M - 1 ? 0 : m + 1;
            v[0] = v[1]; v[1] = v[2]; v[2] = v[3];
            v[3] = r + 4 < N ? __ldcg(x + (long long)(r + 4) * CELLS) : 0.0f;
        }
        return make_double2(ff_value(sum), ff_value(sq));
    }
    for (int r0 = 0; r0 < N; r0 += 8) {
        float v[8];
        const int n = min(8, N - r0);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = q < n ? __ldcg(x + (long long)(r0 + q) * CELLS) : 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (q < n) {
                tally_ray(P, v[q], m, M, &sum, &sq, &rep);
                m = P.sampler && m == M - 1 ? 0 : m + 1;
            }
        }
    }
    return make_double2(ff_value(sum), ff_value(sq));
}

// Dynamic shared memory of a march kernel: a kernel whose static plus
// dynamic shared memory exceeds the default 48 KB per block needs its limit
// raised once (queried first, so a launch inside a graph capture only reads).
inline int march_prepare_smem(void (*k)(const MarchParams), size_t smem) {
    cudaFuncAttributes fa;
    cudaError_t e = cudaFuncGetAttributes(&fa, k);
    if (e != cudaSuccess) return (int)e;
    if (fa.sharedSizeBytes + smem > 48u * 1024u && (size_t)fa.maxDynamicSharedSizeBytes < smem)
        e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return (int)e;
}

// One launch of a march kernel with `smem` bytes of dynamic shared memory,
// and its resident blocks per SM.
inline int march_launch_one(void (*k)(const MarchParams), int blocks, int threads, size_t smem, cudaStream_t st,
                            const MarchParams &p) {
    if (const int e = march_prepare_smem(k, smem)) return e;
    dnsmc::note_launch();
    k<<<blocks, threads, smem, st>>>(p);
    return (int)cudaGetLastError();
}

inline int march_occupancy_one(void (*k)(const MarchParams), int threads, size_t smem) {
    if (march_prepare_smem(k, smem)) return 0;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, threads, smem) != cudaSuccess) return 0;
    return nb;
}

}  // namespace dnsmc
