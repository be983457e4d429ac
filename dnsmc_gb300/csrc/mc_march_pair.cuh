// mc_march_pair.cuh -- the march on the fine grid (the reference's
// kernel_fluid + march_ray, code/mc_gpu.cu:44-438), two cells per lane: the
// absorbing gas with black walls (march_pair_kernel), and the general medium
// with scattering particles and grey walls (march_gen_kernel).
//
// A packet here is 64 cells of one wall-normal plane: tile_a cells along j
// by tile_b = 64 / tile_a along k.  Lane l owns packet cells l and l + 32,
// which share their j index and lie 32 / tile_a rows apart in k.  Every ray
// of the packet shares one direction and one spectral sample, so the voxel
// walk (which face is crossed next, every segment length) is the same for
// all 64 cells: the warp generates it in chunks (walk_chunk), and a lane does
// the per-cell work (field gather, k and Ib lookups, attenuation, tallies).  Every cell's arithmetic is the reference estimator's update
// written with explicit fmaf, and the host replay (oracle/mc_oracle.cpp)
// marches the same 64-cell packets, so it reproduces every cell bit for bit.
//
// march_gen_kernel is the same march for the general medium: absorption
// k + fv a_band and scattering fv s_band per cell; weighted delta tracking
// with a warp-shared decision (q = mean over the packet's live cells of
// fv s_band / majorant, summed by each lane over its cells in order and then
// across lanes; each cell's throughput is multiplied by p / q on a scatter
// and (1 - p) / (1 - q) otherwise, so every cell's expectation is that of
// ordinary delta tracking); Henyey-Greenstein directions; grey diffuse walls.
// Every direction change restarts the walk from the current point.
//
// Its translation units (mc_march_pair.cu, mc_march_gen.cu) are compiled
// with -fmad=false like the other march translation units.
#pragma once
#include "mc_march.cuh"

namespace dnsmc {

// Resident 256-thread blocks per SM of this march (2: up to 128 registers a
// thread; its two cells per lane carry twice the per-cell state).
#ifndef DNSMC_PAIR_MINB
#define DNSMC_PAIR_MINB 2
#endif

// ---------------------------------------------------------------------------
// The walk of a packet-ray, generated by the whole warp.
//
// A walk is the merge of three sorted sequences: the crossing times of the
// wall-normal faces and of the two periodic axes, each a closed form of the
// axis' crossing count (W before A before B where times are equal).  The warp
// generates it in chunks of at most walk_cap steps: the chunk's time window
// is cut into 31 equal slices, lane l starts slice l from the crossing counts
// at the slice's start (closed form, corrected by comparing the very products
// the sequence is made of, so they are exact) and steps through its few
// crossings.  The chunk goes to shared memory as pairs (minus the segment
// length, cell entered two steps later); every lane then reads the same pairs.
// Against computing the walk in every lane beside the attenuation, the step
// loop loses the face choice, the crossing times and the index updates, and
// it knows the cells ahead, so a cell's field value is fetched two steps
// before it is used.
// Marches with the walk in every lane and now: 128^3 correlated-k channel (48
// rays) 85.5 and 61.4 ms (4 of them ray_batch's), grey 64^3 channel at 256 rays
// 9.6 and 2.8 ms.  Chunks of 64 / 96 / 128 / 192 steps: channel 62.5 / 61.9 / 61.6 /
// 61.7 ms (longer chunks take more shared memory a warp).  With uniform
// absorption, and so with 64 wall-normal crossings listed, 128 / 192 / 256: grey
// 2.91 / 2.80 / 2.83, drop-in bands call 6.56 / 6.33 / 6.74 ms.
// ---------------------------------------------------------------------------
// A warp's walk buffer (walk_words): the state after the chunk (8 words), its
// wall-normal times (TIMES + 1, rounded up to 4), then -- the pointer the marches
// hold -- a 4-word header whose last word is the cell entered by the chunk's
// first step, and the pairs (walk_cap, one spare).
__host__ __device__ constexpr int walk_times_words(int times) { return times + 4; }

// the float after a non-negative float
__device__ __forceinline__ float next_up(float v) { return __uint_as_float(__float_as_uint(v) + 1u); }

// crossings of a periodic axis before time tau: the n with (n + off) dt < tau.
// r is an estimate of 1 / dt: its error (a few 2^-24) moves the count by less
// than one up to 2^20 crossings, which one comparison each way mends; larger
// counts (a ray has at most 2^22 steps) are stepped, a bounded number of times
// whatever the inputs.
__device__ __forceinline__ float crossings_before(float tau, float r, float dt, float off) {
    float g = fminf(fmaxf(floorf(fmaf(tau, r, 1.0f - off)), 0.0f), 8388608.0f);
    if (g >= 1048576.0f) {
        for (int i = 0; i < 16 && (g - 1.0f + off) * dt >= tau; ++i) g -= 1.0f;
        for (int i = 0; i < 16 && (g + off) * dt < tau; ++i) g += 1.0f;
    }
    g = (g - 1.0f + off) * dt >= tau ? g - 1.0f : g;
    g = (g + off) * dt < tau ? g + 1.0f : g;
    return g;
}

// v in [0, n) moved by d (any sign) on a periodic axis of n entries
__device__ __forceinline__ int wrap_move(int v, int d, int n) {
    v += d;
    if ((unsigned)v >= (unsigned)n) {
        v = v < 0 ? v + n : v - n;
        if ((unsigned)v >= (unsigned)n) { v %= n; if (v < 0) v += n; }
    }
    return v;
}

struct Walk {
    // the ray: direction signs, the signed inverse of the wall-normal cosine,
    // the times between periodic crossings and estimates of their inverses,
    // the wall-normal start, the periodic start offsets inside the first
    // cell along the direction of travel
    int dW, dA, dB;
    float sinvW, dtA, dtB, rA, rB, oW, offA, offB;
    // state after the steps generated so far: time, crossing counts (as
    // floats: exact, below 2^22), wall-normal cell, the packet corner's
    // periodic cell
    float t, nA, nB;
    int cw, ca, cb;
};

// The ray's direction in the walk, which then starts at time 0 from its
// (oW, offA, offB) offsets.
__device__ __forceinline__ void walk_direction(const MarchParams &P, Walk &w, float sW, float sA, float sB) {
    const float aW = fabsf(sW), aA = fabsf(sA), aB = fabsf(sB);
    const float invW = 1.0f / aW, invA = 1.0f / aA, invB = 1.0f / aB;
    w.dW = sW > 0.f ? 1 : -1; w.dA = sA > 0.f ? 1 : -1; w.dB = sB > 0.f ? 1 : -1;
    // crossing time of a wall-normal face: (fw[c + 1] - o) / s going up,
    // (o - fw[c]) / |s| = (fw[c] - o) * (-1/|s|) going down (exact negation)
    w.sinvW = w.dW > 0 ? invW : -invW;
    w.dtA = P.da * invA; w.dtB = P.db * invB;
    w.rA = aA * P.rda; w.rB = aB * P.rdb;
    w.t = 0.0f; w.nA = 0.0f; w.nB = 0.0f;
}

// How a chunk ends: the walk goes on, its last step reaches a wall, or (COL)
// the tentative collision at time tcol comes next.
enum WalkEnd { WALK_ON = 0, WALK_WALL = 1, WALK_COL = 2 };

// Generate the next chunk (at most cap steps, cap <= walk_cap; about `aim` of
// them; none after tcol).  Returns the steps generated (at least one, but
// before a collision and for unusable faces), *end how the chunk ends.  The
// state is advanced in shared memory (walk_state reads it back; not written
// when there are no steps).
// TIMES (32 or 64): wall-normal crossings a chunk may reach.  64 for uniform
// absorption (rays through all planes take one chunk: grey 64^3 2.90 ms, with 32
// 2.99; drop-in bands call 7.21 and 7.31 ms), 32 for the others (128^3 channel
// 61.6 ms, with 64 62.2; particles at 96^3 11.6 and 12.0 ms).
template <bool TRACE, bool COL, int TIMES>
__device__ __forceinline__ int walk_chunk(const MarchParams &P, const Walk &w, float aim, int cap, float tcol, float *buf,
                                          int lane, int *end, int step0) {
    const unsigned FULL = 0xffffffffu;
    const float INF = __int_as_float(0x7f800000);
    const int dW = w.dW, dA = w.dA, dB = w.dB;
    const float *fwn = P.fw + (dW > 0 ? 1 : 0);
    const float dtA = w.dtA, dtB = w.dtB, rA = w.rA, rB = w.rB;
    float *const tw = buf - walk_times_words(TIMES), *const st = tw - 8;
    // the next TIMES wall-normal crossings
    const int c = w.cw + dW * lane, c2 = c + dW * 32;
    const bool in = (unsigned)c < (unsigned)P.nw, in2 = TIMES > 32 && (unsigned)c2 < (unsigned)P.nw;
    const float twl = in ? (__ldg(fwn + c) - w.oW) * w.sinvW : INF;
    const float twh = in2 ? (__ldg(fwn + c2) - w.oW) * w.sinvW : INF;
    __syncwarp();  // the previous chunk's readers are done
    tw[lane] = twl;
    int nv = __popc(__ballot_sync(FULL, in));                // >= 1: the cell is in the grid
    if (TIMES > 32) {
        tw[32 + lane] = twh;
        nv += __popc(__ballot_sync(FULL, in2));
    }
    const float tw0 = __shfl_sync(FULL, twl, 0), twe = __shfl_sync(FULL, nv > 32 ? twh : twl, (nv - 1) & 31);
    if (lane == 0) {
        tw[TIMES] = INF;
        st[6] = 0.0f;  // (int) 0 steps, unless a lane makes the last one
    }
    // the window: about `aim` crossings at the present rates, no more than
    // the listed wall-normal ones, at least the next crossing
    const float rW = twe < INF ? __fdividef((float)(nv - 1), fmaxf(twe - tw0, 1e-30f)) : 0.0f;
    float te = w.t + __fdividef(aim, rA + rB + rW);
    te = fminf(te, nv < TIMES ? (twe < INF ? next_up(twe) : INF) : twe);
    const float tmin = fminf(tw0, fminf((w.nA + w.offA) * dtA, (w.nB + w.offB) * dtB));
    te = fmaxf(te, next_up(tmin));
    bool col = false;
    if (COL && tcol < INF) {
        const float tc = next_up(tcol);
        col = tc <= te;
        te = fminf(te, tc);
    }
    const float dt = (te - w.t) * (1.0f / 31.0f);
    const float tau = lane == 31 ? te : fminf(fmaf((float)lane, dt, w.t), te);
    // crossing counts at this lane's slice start
    float nA = w.nA, nB = w.nB;
    int k = 0;
    __syncwarp();
    if (lane) {
        nA = fmaxf(nA, crossings_before(tau, rA, dtA, w.offA));
        nB = fmaxf(nB, crossings_before(tau, rB, dtB, w.offB));
#pragma unroll
        for (int h = TIMES / 2; h; h >>= 1) k += tw[k + h - 1] < tau ? h : 0;
        k += tw[k] < tau ? 1 : 0;
    }
    const int mA = (int)(nA - w.nA), mB = (int)(nB - w.nB);
    int e = mA + mB + k;
    const int total = __shfl_sync(FULL, e, 31);
    const int eend = min(__shfl_down_sync(FULL, e, 1), cap);
    const int n0 = min(total, cap);
    bool hit = false;
    if (lane < 31 && e < eend) {
        // (the bounds hold by themselves for faces in ascending order)
        int cw = min(max(w.cw + dW * k, 0), P.nw - 1), ca = wrap_move(w.ca, dA * mA, P.na), cb = wrap_move(w.cb, dB * mB, P.nb);
        float tA = (nA + w.offA) * dtA, tB = (nB + w.offB) * dtB, tW = tw[k];
        // the time of the crossing before the slice
        float t = fmaxf(w.t, fmaxf((nA - 1.0f + w.offA) * dtA, (nB - 1.0f + w.offB) * dtB));
        if (k) t = fmaxf(t, tw[k - 1]);
        int off = (int)(((unsigned)cw * P.pnb + cb) * P.pna + ca);
        do {
            const bool bW = tW <= tA && tW <= tB;
            const bool bA = !bW && tA <= tB;
            const float tn = bW ? tW : (bA ? tA : tB);
            if (TRACE && step0 + e < P.trace_max) {
                int *rec = P.trace_rec + 6 * (step0 + e);
                rec[0] = cw; rec[1] = dA * (int)nA; rec[2] = dB * (int)nB; rec[3] = bW ? 0 : (bA ? 1 : 2);
                rec[4] = __float_as_int(tn - t);
            }
            buf[4 + 2 * e] = t - tn;
            t = tn;
            if (bW) {
                hit = (unsigned)(cw + dW) >= (unsigned)P.nw;
                if (!hit) { cw += dW; k = min(k + 1, TIMES); tW = tw[k]; }
            } else if (bA) {
                nA += 1.0f;
                tA = (nA + w.offA) * dtA;
                ca += dA;
                ca = ca == P.na ? 0 : (ca < 0 ? P.na - 1 : ca);
            } else {
                nB += 1.0f;
                tB = (nB + w.offB) * dtB;
                cb += dB;
                cb = cb == P.nb ? 0 : (cb < 0 ? P.nb - 1 : cb);
            }
            off = (int)(((unsigned)cw * P.pnb + cb) * P.pna + ca);
            buf[3 + 2 * e] = __int_as_float(off);
            ++e;
        } while (e < eend && !hit);
        if (e == n0 || hit) {  // this lane made the chunk's last step: the state, and the spare pairs
            st[0] = t; st[1] = nA; st[2] = nB;
            st[3] = __int_as_float(cw); st[4] = __int_as_float(ca); st[5] = __int_as_float(cb);
            st[6] = __int_as_float(e);
            buf[4 + 2 * e] = 0.0f;             // a pair of zero length: changes nothing
            buf[3 + 2 * e] = __int_as_float(off);
            buf[5 + 2 * e] = __int_as_float(off);
        }
    }
    hit = __any_sync(FULL, hit);
    *end = hit ? WALK_WALL : (col && total <= cap ? WALK_COL : WALK_ON);
    __syncwarp();
    return __float_as_int(st[6]);
}

template <int TIMES>
__device__ __forceinline__ void walk_state(const float *buf, Walk &w) {
    const float *st = buf - walk_times_words(TIMES) - 8;
    w.t = st[0]; w.nA = st[1]; w.nB = st[2];
    w.cw = __float_as_int(st[3]); w.ca = __float_as_int(st[4]); w.cb = __float_as_int(st[5]);
}

// A batch of an item's rays, set up a lane each: words, direction, spectral
// sample and (control variate) the surrogate of ray r0 + lane go to shared
// memory, from where the warp takes them ray by ray.
// Every lane setting up every ray took 250 of its ~3000 instructions (128^3
// channel 66.1 ms, so 62.3; 4 x 96^3 batch 130.1 and 119.6 ms).
struct RayBatch {
    float4 walk[32];    // sinvW, dtA and dtB (signed like the direction; general medium: the
                        // direction itself), the sample's weight factor
    float4 rates[32];   // rA, rB, band and spectral sample (as int bits)
    float4 sur[32];     // surrogate: collected intensity, own-layer absorptance, own-layer intensity
};
static_assert(sizeof(RayBatch) == kBatchBytes, "march_pair_smem");

template <int MODE, bool TRACE, bool CV, bool GEN>
__device__ __forceinline__ void ray_batch(const MarchParams &P, RayBatch *B, int r, int M, int p, uint32_t ctr2, int gs,
                                         int K, int f, int w0, int lane) {
    uint4 x;
    if (P.sampler) {
        const int b = r / M;
        const uint4 sh = philox4x32_10(make_uint4((uint32_t)b, (uint32_t)p, ctr2, 0x50B01u), P.key0, P.key1);
        const uint4 sb = sobol4((uint32_t)(r - b * M));
        x = make_uint4(sb.x ^ sh.x, sb.y ^ sh.y, sb.z ^ sh.z, sb.w ^ sh.w);
    } else {
        x = philox4x32_10(make_uint4((uint32_t)r, (uint32_t)p, ctr2, 0u), P.key0, P.key1);
    }
    if (TRACE && lane == 0) {
        P.trace_rng[0] = x.x; P.trace_rng[1] = x.y; P.trace_rng[2] = x.z; P.trace_rng[3] = x.w;
    }
    float sW, sA, sB;
    ray_direction(x, &sW, &sA, &sB);
    Walk w;
    walk_direction(P, w, sW, sA, sB);
    float eW = P.Wgrey;
    int nbnd = 0, sid = 0;
    if constexpr (MODE != MODE_GREY) {
        const int j = (int)__umulhi(x.z, (uint32_t)K);
        SpecEntry e = P.entries[gs + j];
        if (!(u24(x.w) < e.prob)) e = P.entries[gs + (int)(e.alias_nb & 0xFFFFu)];
        nbnd = (int)(e.alias_nb >> 16);
        sid = e.koff;
        eW = e.W;
    }
    B->walk[lane] = GEN ? make_float4(sW, sA, sB, eW)
                        : make_float4(w.sinvW, w.dA > 0 ? w.dtA : -w.dtA, w.dB > 0 ? w.dtB : -w.dtB, eW);
    B->rates[lane] = make_float4(w.rA, w.rB, __int_as_float(nbnd), __int_as_float(sid));
    if (CV) {
        // the ray's straight flight through the layer-mean medium, the same
        // for all cells (same layer)
        const long long srow = ((long long)f * P.n_samples + sid) * P.nw + w0;
        float J, A;
        surrogate_lookup(P.surtab + srow * (2 * kSurBins), sW, &J, &A);
        B->sur[lane] = make_float4(J, A, __ldg(P.sur + srow).y, 0.0f);
    }
}

// Field values of the march on the fine grid: [f][i][k][j] of rows of pna
// values, pnb rows a plane: the periodic axes continue past their end by the
// packet's extent, so a lane's cells lie at fixed offsets from the packet's
// corner wherever the walk has moved it.
template <int MODE, bool UNI> struct PairFieldT { typedef typename FieldT<MODE>::type type; };
template <> struct PairFieldT<MODE_T, true> { typedef float type; };  // the table coordinate
template <int MODE, bool UNI>
__device__ __forceinline__ const typename PairFieldT<MODE, UNI>::type *field_base(const MarchParams &P) {
    if constexpr (MODE == MODE_TX) return P.fieldPX;
    else if constexpr (MODE == MODE_T && UNI) return P.fieldF;
    else if constexpr (MODE == MODE_T) return P.fieldP;
    else return P.fieldG;
}

// Ib from clamped table coordinates p (uniform absorption: nothing else is
// looked up).  Adding 2^23 rounded down leaves floor(p) in the low bits of the
// sum, which the address of the slab's entry takes as it is; the entry past
// the last cell is the end point's value.  Split as pos_split, bit for bit,
// the lane's two cells in paired instructions.  4 bytes a cell instead of (index, fraction): the L1 data
// pipe bounded the band tables' march (86 %), and a gather of 32 four-byte cells takes 2 of
// its cycles instead of 4.2: drop-in bands call 7.17 -> 6.74 ms.
struct SlabIb {
    // addresses of the slab and of its Ib part, less the bits of 2^23 (with the
    // slab's held too the compiler takes one instruction less a lookup: 6.74 -> 6.55 ms)
    unsigned slab, ia;
    __device__ __forceinline__ SlabIb(const float2 *slk, const float2 *sli)
        : slab(smem_addr(slk) - 0x4B000000u * 8u), ia(smem_addr(sli) - 0x4B000000u * 8u) {}
    // once a ray's slab has arrived: no lookup of it may move ahead
    __device__ __forceinline__ void arrived() { asm volatile("" : "+r"(slab), "+r"(ia)::"memory"); }
    __device__ __forceinline__ static float entry(unsigned at, float f) {
        float a, d;
        asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(d) : "r"(at));
        return fmaf(f, d, a);
    }
    __device__ __forceinline__ float2 lookup(float2 p) const {
        const float2 sh = make_float2(8388608.0f, 8388608.0f);
        const float2 s = __fadd2_rd(p, sh);
        const float2 f = __fadd2_rn(p, __ffma2_rn(s, make_float2(-1.0f, -1.0f), sh));
        return make_float2(entry(__float_as_uint(s.x) * 8u + ia, f.x), entry(__float_as_uint(s.y) * 8u + ia, f.y));
    }
};

// Resident 256-thread blocks per SM.  Tables: 2 (128 registers: the values of
// four steps of two cells; 3 spill, 66.2 -> 70.1 ms on the 128^3 channel).
// UNI: 4 (64 registers): its steps are short, so the walk's generation and the
// gathers need more warps to hide behind -- grey 64^3 4.00 (2) / 3.12 (3) / 2.99
// ms (4), grey bands through the drop-in pair 8.34 / 7.59 / 7.29 ms.  Moments (18
// FP64 sums a lane): 2.
__host__ __device__ constexpr int pair_min_blocks(bool uni, bool mom) {
    return uni && !mom ? 4 : DNSMC_PAIR_MINB;
}

// UNI: the absorption coefficient is the same everywhere (grey model, grey
// band tables), so are a step's attenuation and the packet's transmissivity:
// the warp computes expm1 of a chunk's steps side by side, a cell-step is one
// gather, one difference and one fused multiply-add.  SPLIT: items in
// several queue units (MarchParams::parts).
template <int MODE, bool UNI, bool TRACE, bool CV, bool MOM, bool SPLIT>
__global__ void __launch_bounds__(256, pair_min_blocks(UNI, MOM)) march_pair_kernel(const MarchParams P) {
    typedef typename PairFieldT<MODE, UNI>::type VT;
    constexpr bool BANDS = MODE == MODE_T && UNI;
    constexpr int C = kLaneCells;  // cells per lane
    static_assert(C == 2, "the attenuation goes through a cell pair");
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int tid = threadIdx.x;
    const int la = lane % P.tile_a, lb = lane / P.tile_a;
    const int hb = 32 / P.tile_a;  // k rows between a lane's two cells
    const int njR = P.ea1 - P.ea0, nkR = P.eb1 - P.eb0;
    unsigned long long my_rays = 0, my_steps = 0;
    unsigned int flags = 0;
    // dynamic shared memory (march_pair_smem): this warp's copy of the
    // current ray's table slab (tabulated models), its walk buffer and ray batch;
    // per-cell sums of the item as float pairs (ray sum, sum of squares or of
    // squared replicate means, current replicate sum) [3][C][threads] --
    // shared memory, so registers hold the march's own working set
    extern __shared__ float4 s_dyn[];
    const int nthr = blockDim.x;
    const int warp = threadIdx.x >> 5, nwarp = (nthr + 31) >> 5;
    float2 *const slk = reinterpret_cast<float2 *>(s_dyn) + warp * P.slab_len;
    const float2 *const sli = slk + P.slab_klen;
    float *const wbuf = reinterpret_cast<float *>(reinterpret_cast<float2 *>(s_dyn) + nwarp * P.slab_len) + warp * walk_words(UNI) + 8 + walk_times_words(UNI ? 64 : 32);
    RayBatch *const batch = reinterpret_cast<RayBatch *>(reinterpret_cast<float *>(reinterpret_cast<float2 *>(s_dyn) + nwarp * P.slab_len) +
                                                        nwarp * walk_words(UNI)) + warp;
    float2 *const s_acc = reinterpret_cast<float2 *>(batch - warp + nwarp);
    auto acc = [&](int q, int k) { return s_acc + (q * C + k) * nthr + tid; };
    // each warp's transaction barrier of its slab copies, and its parity
    __shared__ uint64_t s_bar[8];
    uint64_t *const sbar = &s_bar[warp];
    uint32_t sphase = 0;
    slab_bar_init(sbar, lane);
    SlabIb tib(slk, sli);
    bool dead = false;  // a slab copy did not arrive: this warp stops marching

    for (;;) {
        long long item;  // below 2^32, as the queue
        int part = 0;
        if (TRACE) {
            if (threadIdx.x >= 32) return;
            item = ((long long)P.trace_f * P.n_groups + P.trace_g) * P.n_packets + P.trace_p;
        } else {
            unsigned int it = 0;
            if (lane == 0) it = atomicAdd(P.queue, 1u);
            it = __shfl_sync(FULL, it, 0);
            if ((long long)it >= (SPLIT ? P.n_items * P.parts : P.n_items)) break;
            if (SPLIT) {
                part = (int)(it % (unsigned)P.parts);
                it /= (unsigned)P.parts;
            }
            item = P.item_order ? (long long)__ldg(P.item_order + it) : (long long)it;
        }
        const unsigned fg = (unsigned)item / (unsigned)P.n_packets;
        const int p = (int)((unsigned)item - fg * (unsigned)P.n_packets);
        const int f = (int)(fg / (unsigned)P.n_groups), G = (int)(fg - (unsigned)f * (unsigned)P.n_groups);
        const int pa = p % P.npa;
        const int rest = p / P.npa;
        const int pb = rest % P.npb;
        const int pw = rest / P.npb;
        const int w0 = P.ew0 + pw;
        const int ac = P.ea0 + pa * P.tile_a, bc = P.eb0 + pb * P.tile_b;  // the packet's corner
        bool active[C];
        int tcell[C];
        const VT *fp[C];  // the lane's cells as offsets from the corner (cells outside the region: the corner)
#pragma unroll
        for (int k = 0; k < C; ++k) {
            active[k] = ac + la < P.ea1 && bc + lb + k * hb < P.eb1;
            const int a = active[k] ? la : 0, b = active[k] ? lb + k * hb : 0;
            tcell[k] = (pw * nkR + pb * P.tile_b + b) * njR + pa * P.tile_a + a;
            fp[k] = field_base<MODE, UNI>(P) + (long long)f * P.pstride + b * P.pna + a;
        }
        const unsigned corner = ((unsigned)w0 * P.pnb + bc) * P.pna + ac;
        const int N = P.rays_per_packet ? P.rays_per_packet[G * P.rays_gstride + p] : P.rays;
        const float oW = (__ldg(P.fw + w0) + __ldg(P.fw + w0 + 1)) * 0.5f;
        // alias table of this packet: band group G of the temperature bin
        // nearest to the temperature of the packet's first cell
        int gs = 0, K = 1;
        if constexpr (MODE == MODE_GREY) {
            // T^4 with the sign set where the temperature is not positive
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const float v = __ldg(fp[k] + corner);
                if (active[k] && (__float_as_int(v) < 0 || v != v)) flags |= DNSMC_STATUS_BAD_FIELD;
            }
        } else {
            int boff = 0;
            if (P.n_tbins > 1) {
                float tp;
                if constexpr (BANDS) {
                    tp = __ldg(fp[0] + corner);
                } else {
                    int kx, ti;
                    float ft, fx;
                    cell_coords<MODE>(__ldg(fp[0] + corner), &kx, &ti, &ft, &fx);
                    tp = (float)ti + ft;
                }
                const float tp0 = __shfl_sync(FULL, tp, 0);
                int bin = __float2int_rn(tp0);
                bin = min(max(bin, 0), P.n_tbins - 1);
                boff = bin * P.n_groups;
            }
            gs = P.group_start[boff + G];
            K = P.group_start[boff + G + 1] - gs;
        }
        const uint32_t ctr2 = (uint32_t)G | ((uint32_t)(f + P.field_base) << 16);
        double mo[C][9];
        if (MOM)
#pragma unroll
            for (int k = 0; k < C; ++k)
#pragma unroll
                for (int q = 0; q < 9; ++q) mo[k][q] = 0.0;
        const int M = P.sampler ? max(1, N / max(1, P.nbatch)) : 1;
        if (!SPLIT)
#pragma unroll
        for (int k = 0; k < C; ++k) {
            *acc(0, k) = make_float2(0.0f, 0.0f); *acc(1, k) = make_float2(0.0f, 0.0f); *acc(2, k) = make_float2(0.0f, 0.0f);
        }
        unsigned long long isteps = 0;
        unsigned int lsteps = 0;  // this lane's active cell-steps in the item
        int rbeg = TRACE ? P.trace_r : 0;
        int rend = TRACE ? P.trace_r + 1 : ((K > 0) ? N : 0);
        float *const rayx = SPLIT ? P.rayx + item * N * 64 + lane : nullptr;
        if (SPLIT) unit_rays(P, part, rend, &rbeg, &rend);
        int m = P.sampler ? rbeg % M : 0;  // the ray's index in its replicate
        int est = 32;                      // steps of a ray of this item, a running mean
        for (int r = rbeg; r < rend; ++r) {
            const int rb = (r - rbeg) & 31;
            if (rb == 0) {
                __syncwarp();
                if (r + lane < rend) ray_batch<MODE, TRACE, CV, false>(P, batch, r + lane, M, p, ctr2, gs, K, f, w0, lane);
                __syncwarp();
            }
            // the ray's table slab is on its way while the walk's first chunk
            // is generated
            const float4 bw = batch->walk[rb], br = batch->rates[rb];
            if constexpr (MODE != MODE_GREY) slab_issue(P, __float_as_int(br.w), smem_addr(slk), lane, sbar);
            Walk w;
            w.dW = bw.x > 0.0f ? 1 : -1; w.dA = bw.y > 0.0f ? 1 : -1; w.dB = bw.z > 0.0f ? 1 : -1;
            w.sinvW = bw.x; w.dtA = fabsf(bw.y); w.dtB = fabsf(bw.z);
            w.rA = br.x; w.rB = br.y;
            w.oW = oW; w.offA = 0.5f; w.offB = 0.5f;
            w.t = 0.0f; w.nA = 0.0f; w.nB = 0.0f;
            w.cw = w0; w.ca = ac; w.cb = bc;
            VT va[C], vb[C], vc[C], vd[C];  // field values of two steps and of the two after
#pragma unroll
            for (int k = 0; k < C; ++k) va[k] = __ldg(fp[k] + corner);
            float wk[C], Ii[C], tau[C], D[C];
            // the step at which each cell was dumped (its live steps are that
            // plus one; cells never dumped were live for every step)
            int life[C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                tau[k] = UNI || active[k] ? 1.0f : 0.0f;
                D[k] = 0.0f;
                life[k] = 1 << 30;
            }
            int steps = 0;
            bool first = true;
            for (;;) {  // chunks of the walk
                int end;
                // a short first chunk where this item's rays have been short
                const int n = walk_chunk<TRACE, false, UNI ? 64 : 32>(P, w, first && est < 20 ? 28.0f : (float)(walk_cap(UNI) - 4),
                                                       min(walk_cap(UNI), P.max_steps - steps), 0.0f, wbuf, lane, &end, steps);
                if constexpr (UNI) {
                    // e = expm1(k (t - tn)) of the chunk's steps, a lane each
                    for (int q = lane; q < n; q += 32) wbuf[4 + 2 * q] = mc_expm1(P.kappa * wbuf[4 + 2 * q]);
                    __syncwarp();
                }
                {
                    const unsigned c1 = n ? __float_as_uint(wbuf[3]) : corner;
#pragma unroll
                    for (int k = 0; k < C; ++k) vb[k] = __ldg(fp[k] + c1);
                }
                if (first) {
                    first = false;
                    if constexpr (MODE != MODE_GREY)
                        if (!slab_wait(P, sbar, &sphase, &flags)) { dead = true; break; }
                    if constexpr (BANDS) {
                        tib.arrived();
                        const float2 ib = tib.lookup(make_float2(va[0], va[1]));
                        Ii[0] = ib.x; Ii[1] = ib.y;
                    }
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        if constexpr (MODE == MODE_GREY) {
                            Ii[k] = va[k];
                            wk[k] = bw.w;
                        } else if constexpr (BANDS) {
                            wk[k] = bw.w * P.kappa;
                        } else {
                            int kx, ti;
                            float ft, fx;
                            cell_coords<MODE>(va[k], &kx, &ti, &ft, &fx);
                            const float ki = lookup_k<MODE>(slk, kx, ft, fx);
                            Ii[k] = lookup_ib(sli, ti, ft);
                            wk[k] = bw.w * ki;
                        }
                    }
                }
                if (n == 0) {  // no walk through these faces (not in ascending order, or not finite)
                    flags |= DNSMC_STATUS_STEP_CAP;
                    break;
                }
                const float4 *wp = reinterpret_cast<const float4 *>(wbuf + 4);
                bool done = false;
                // One step.  Per cell: alpha = -expm1(-k ds), ta = tau alpha,
                // D += ta g, tau -= ta, with g = Ii - Ib_j: D is the net
                // exchange in intensity units and the ray's contribution wk D
                // (the reference normalises g by Ii and multiplies the ray by
                // Ii again).  A cell already dumped (tau 0) adds exactly
                // nothing.  The two cells of the pair go through paired FP32
                // instructions with every sign moved onto an operand whose
                // negation is exact: e = expm1(k * (t - tn)) = -alpha, nta =
                // tau e = -ta, D += nta (-g), tau += nta -- the same roundings.
                auto neg_g = [&](const VT (&v)[C]) {  // UNI: -g of the cells
                    if constexpr (MODE == MODE_GREY) {
                        return make_float2(v[0] - Ii[0], v[1] - Ii[1]);
                    } else if constexpr (BANDS) {
                        const float2 ib = tib.lookup(make_float2(v[0], v[1]));
                        return make_float2(ib.x - Ii[0], ib.y - Ii[1]);
                    } else {
                        return make_float2(0.0f, 0.0f);
                    }
                };
                auto step = [&](const VT (&v)[C], float nds, int s) {
                    if constexpr (UNI) {
                        const float nta = tau[0] * nds;  // nds: expm1 of the step
                        const float2 g = neg_g(v);
                        const float ng[C] = {g.x, g.y};
#pragma unroll
                        for (int k = 0; k < C; ++k) D[k] = fmaf(nta, ng[k], D[k]);
                        tau[0] = tau[0] + nta;
                        if (TRACE && lane == 0 && s < P.trace_max)
                            P.trace_rec[6 * s + 5] = __float_as_int(tau[0] < P.toll ? 0.0f : tau[0]);
                        if (tau[0] < P.toll) {  // the same in every lane
#pragma unroll
                            for (int k = 0; k < C; ++k) D[k] = fmaf(-tau[0], ng[k], D[k]);
                            tau[0] = 0.0f;
                            life[0] = life[1] = s;
                            done = true;
                        }
                    } else {
                        float kj[C], ngj[C];
#pragma unroll
                        for (int h = 0; h < C; ++h) {
                            int kx, tj;
                            float ftj, fxj;
                            cell_coords<MODE>(v[h], &kx, &tj, &ftj, &fxj);
                            kj[h] = lookup_k<MODE>(slk, kx, ftj, fxj);
                            const float Ibj = lookup_ib(sli, tj, ftj);
                            ngj[h] = Ibj - Ii[h];
                        }
                        const float2 e = mc_expm1_x2(__fmul2_rn(make_float2(kj[0], kj[1]), make_float2(nds, nds)));
                        const float2 nta = __fmul2_rn(make_float2(tau[0], tau[1]), e);
                        const float2 d2 = __ffma2_rn(nta, make_float2(ngj[0], ngj[1]), make_float2(D[0], D[1]));
                        const float2 t2 = __fadd2_rn(make_float2(tau[0], tau[1]), nta);
                        D[0] = d2.x; D[1] = d2.y;
                        tau[0] = t2.x; tau[1] = t2.y;
#pragma unroll
                        for (int h = 0; h < C; ++h) {
                            if (tau[h] < P.toll) {
                                D[h] = fmaf(-tau[h], ngj[h], D[h]);
                                tau[h] = 0.0f;
                                life[h] = min(life[h], s);
                            }
                        }
                        if (TRACE && lane == 0 && s < P.trace_max) P.trace_rec[6 * s + 5] = __float_as_int(tau[0]);
                    }
                };
                // Two steps on v0, v1 while the two after are fetched into v2,
                // v3; the warp's exit vote after the second (a walk may then
                // take one step past the one that dumped its last live cell,
                // which changes nothing).
                float4 wc = wp[0];
                int s = 0;
                auto pair = [&](const VT (&v0)[C], const VT (&v1)[C], VT (&v2)[C], VT (&v3)[C]) {
                    const unsigned o2 = __float_as_uint(wc.y), o3 = __float_as_uint(wc.w);
#pragma unroll
                    for (int k = 0; k < C; ++k) v2[k] = __ldg(fp[k] + o2);
#pragma unroll
                    for (int k = 0; k < C; ++k) v3[k] = __ldg(fp[k] + o3);
                    const float d0 = wc.x, d1 = wc.z;
                    wc = *++wp;
                    if constexpr (UNI && !TRACE) {
                        // the two steps at once unless one of them ends the ray (the
                        // checks of both in one branch: grey 64^3 3.39 -> 3.12 ms)
                        const float n0 = tau[0] * d0, t0 = tau[0] + n0, n1 = t0 * d1, t1 = t0 + n1;
                        if (t0 >= P.toll && t1 >= P.toll) {
                            const float2 g0 = neg_g(v0), g1 = neg_g(v1);
                            D[0] = fmaf(n1, g1.x, fmaf(n0, g0.x, D[0]));
                            D[1] = fmaf(n1, g1.y, fmaf(n0, g0.y, D[1]));
                            tau[0] = t1;
                            s += 2;
                            return;
                        }
                    }
                    step(v0, d0, steps + s);
                    if (UNI && done) return;
                    step(v1, d1, steps + s + 1);
                    if constexpr (!UNI) done = !__any_sync(FULL, !(tau[0] < P.toll) || !(tau[1] < P.toll));
                    s += 2;
                };
                for (;;) {
                    pair(va, vb, vc, vd);
                    if (done || s >= n) break;
                    pair(vc, vd, va, vb);
                    if (done || s >= n) break;
                }
                if (done) { steps += n; break; }
                steps += n;
                if (end == WALK_WALL) {
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const int side = w.dW > 0 ? 1 : 0;
                        const float Iw = (MODE == MODE_GREY) ? P.Tw4[side] : __ldg(P.ibw + side * P.nbands + __float_as_int(br.z));
                        D[k] = fmaf(UNI ? tau[0] : tau[k], Ii[k] - Iw, D[k]);
                    }
                    break;
                }
                if (steps >= P.max_steps) {
                    if (UNI ? (active[0] || active[1]) : (!(tau[0] < P.toll) || !(tau[1] < P.toll)))
                        flags |= DNSMC_STATUS_STEP_CAP;
                    break;
                }
                walk_state<UNI ? 64 : 32>(wbuf, w);
                {  // the cell the next chunk starts in
                    const unsigned c0 = ((unsigned)w.cw * P.pnb + w.cb) * P.pna + w.ca;
#pragma unroll
                    for (int k = 0; k < C; ++k) va[k] = __ldg(fp[k] + c0);
                }
            }
            if (dead) break;
            {
                // the walk's length: the step that dumped the last live cell
                // plus one (never dumped: every generated step)
                int last = max(life[0], life[1]);
                if constexpr (!UNI) last = __reduce_max_sync(FULL, last);
                steps = min(steps, last + 1);
                est += (min(steps, 128) - est) / 4;
            }
            if (TRACE && lane == 0) *P.trace_n = steps;
#pragma unroll
            for (int k = 0; k < C; ++k) lsteps += active[k] ? (unsigned)min(life[k] + 1, steps) : 0u;
            isteps += (unsigned long long)steps;
            const float4 sur = CV ? batch->sur[rb] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                float X = wk[k] * D[k];
                if (CV) {
                    // Y_a: the ray through the layer-mean medium; Y_b: its own-layer part
                    const float Ya = wk[k] * (Ii[k] - sur.x);
                    const float Yb = wk[k] * (sur.y * (Ii[k] - sur.z));
                    if (MOM && active[k]) {
                        const double xd = X, ya = Ya, yb = Yb;
                        mo[k][0] += xd; mo[k][1] += ya; mo[k][2] += yb;
                        mo[k][3] = fma(xd, xd, mo[k][3]); mo[k][4] = fma(ya, ya, mo[k][4]);
                        mo[k][5] = fma(yb, yb, mo[k][5]); mo[k][6] = fma(xd, ya, mo[k][6]);
                        mo[k][7] = fma(xd, yb, mo[k][7]); mo[k][8] = fma(ya, yb, mo[k][8]);
                    }
                    const float2 beta = P.beta ? P.beta[fg * P.region_cells + tcell[k]] : make_float2(1.0f, -1.0f);
                    X = X - beta.x * Ya;  // tallied: X - beta_a Y_a - beta_b Y_b; the
                    X = X - beta.y * Yb;  // means beta . E[Y] are added back at finalize
                }
                if (active[k]) {
                    ++my_rays;
                    if (!isfinite(X)) flags |= DNSMC_STATUS_NONFINITE;
                    if (SPLIT) rayx[(long long)r * 64 + 32 * k] = X;
                    else tally_ray(P, X, m, M, acc(0, k), acc(1, k), acc(2, k));
                }
            }
            m = P.sampler && m == M - 1 ? 0 : m + 1;
        }
        if (dead) break;  // the item's sums are incomplete; the solve fails
        my_steps += lsteps;
        if (TRACE) return;
        if (SPLIT) {
            if (P.item_steps && lane == 0) atomicAdd(P.item_steps + item, isteps);
            if (unit_done(P, item, lane)) {
#pragma unroll
                for (int k = 0; k < C; ++k)
                    if (active[k]) P.tally[fg * P.region_cells + tcell[k]] = sum_rays<64>(P, rayx + 32 * k, K > 0 ? N : 0, M);
            }
            continue;
        }
        if (P.item_steps && lane == 0) P.item_steps[item] = isteps;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            if (!active[k]) continue;
            const long long o = fg * P.region_cells + tcell[k];
            P.tally[o] = make_double2(ff_value(*acc(0, k)), ff_value(*acc(1, k)));
            if (MOM) {
                double *out = P.moments + o * 9;
#pragma unroll
                for (int q = 0; q < 9; ++q) out[q] = mo[k][q];
            }
        }
    }
    if (dead) slab_drain(sbar, sphase);
    // per-warp counters and status
    for (int o = 16; o > 0; o >>= 1) {
        my_rays += __shfl_xor_sync(FULL, my_rays, o);
        my_steps += __shfl_xor_sync(FULL, my_steps, o);
        flags |= __shfl_xor_sync(FULL, flags, o);
    }
    if (lane == 0) {
        if (my_rays) atomicAdd(P.counters + 0, my_rays);
        if (my_steps) atomicAdd(P.counters + 1, my_steps);
        if (flags) atomicOr(P.status, flags);
    }
}

// ---------------------------------------------------------------------------
// The same march for the general medium (GEN): particles with scattering and
// grey diffuse walls.  The walk restarts at every scattering and wall
// reflection; its chunks end at the ray's next tentative collision, which is a
// step of its own.
// It is bound by issue and instruction fetches (each collision runs long straight
// code); a cell's volume fraction rides in its 16-byte coordinates, and the
// collisions' random words, free paths and angles are set up a lane each.  96^3
// gas with particles, 8 rays: 10.95 ms (19.8 with the walk in every lane, 0.4
// more with the events' set-up in every lane).
// ---------------------------------------------------------------------------
constexpr int kEvents = 16;  // a batch of a ray's collision and reflection events
static_assert(kEvents * 2 * sizeof(float4) == kEventBytes, "march_pair_smem");
template <int MODE> struct GenFieldT { typedef int4 type; };
template <> struct GenFieldT<MODE_GREY> { typedef float2 type; };
__device__ __forceinline__ float gen_fraction(const int4 &v) { return __int_as_float(v.w); }
__device__ __forceinline__ float gen_fraction(const float2 &v) { return v.y; }

template <int MODE, bool TRACE, bool CV, bool MOM, bool SPLIT>
__global__ void __launch_bounds__(256, DNSMC_PAIR_MINB) march_gen_kernel(const MarchParams P) {
    typedef typename GenFieldT<MODE>::type VT;
    const float INF = __int_as_float(0x7f800000);
    constexpr int C = kLaneCells;  // cells per lane
    static_assert(C == 2, "the attenuation goes through a cell pair");
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int tid = threadIdx.x;
    const int la = lane % P.tile_a, lb = lane / P.tile_a;
    const int hb = 32 / P.tile_a;  // k rows between a lane's two cells
    const int njR = P.ea1 - P.ea0, nkR = P.eb1 - P.eb0;
    unsigned long long my_rays = 0, my_steps = 0;
    unsigned int flags = 0;
    // dynamic shared memory as the gas march's (march_pair_smem)
    extern __shared__ float4 s_dyn[];
    const int nthr = blockDim.x;
    const int warp = threadIdx.x >> 5, nwarp = (nthr + 31) >> 5;
    float2 *const slk = reinterpret_cast<float2 *>(s_dyn) + warp * P.slab_len;
    const float2 *const sli = slk + P.slab_klen;
    float *const wbuf = reinterpret_cast<float *>(reinterpret_cast<float2 *>(s_dyn) + nwarp * P.slab_len) + warp * walk_words(false) + 8 + walk_times_words(32);
    RayBatch *const batch = reinterpret_cast<RayBatch *>(reinterpret_cast<float *>(reinterpret_cast<float2 *>(s_dyn) + nwarp * P.slab_len) +
                                                        nwarp * walk_words(false)) + warp;
    float4 *const events = reinterpret_cast<float4 *>(batch - warp + nwarp) + warp * 2 * kEvents;
    float2 *const s_acc = reinterpret_cast<float2 *>(events + (nwarp - warp) * 2 * kEvents);
    auto acc = [&](int q, int k) { return s_acc + (q * C + k) * nthr + tid; };
    // each warp's transaction barrier of its slab copies, and its parity
    __shared__ uint64_t s_bar[8];
    uint64_t *const sbar = &s_bar[warp];
    uint32_t sphase = 0;
    slab_bar_init(sbar, lane);
    uint32_t slab = smem_addr(slk);
    asm volatile("" : "+r"(slab));  // held, not computed again for every ray
    bool dead = false;  // a slab copy did not arrive: this warp stops marching

    for (;;) {
        long long item;  // below 2^32, as the queue
        int part = 0;
        if (TRACE) {
            if (threadIdx.x >= 32) return;
            item = ((long long)P.trace_f * P.n_groups + P.trace_g) * P.n_packets + P.trace_p;
        } else {
            unsigned int it = 0;
            if (lane == 0) it = atomicAdd(P.queue, 1u);
            it = __shfl_sync(FULL, it, 0);
            if ((long long)it >= (SPLIT ? P.n_items * P.parts : P.n_items)) break;
            if (SPLIT) {
                part = (int)(it % (unsigned)P.parts);
                it /= (unsigned)P.parts;
            }
            item = P.item_order ? (long long)__ldg(P.item_order + it) : (long long)it;
        }
        const unsigned fg = (unsigned)item / (unsigned)P.n_packets;
        const int p = (int)((unsigned)item - fg * (unsigned)P.n_packets);
        const int f = (int)(fg / (unsigned)P.n_groups), G = (int)(fg - (unsigned)f * (unsigned)P.n_groups);
        const int pa = p % P.npa;
        const int rest = p / P.npa;
        const int pb = rest % P.npb;
        const int pw = rest / P.npb;
        const int w0 = P.ew0 + pw;
        const int ac = P.ea0 + pa * P.tile_a, bc = P.eb0 + pb * P.tile_b;  // the packet's corner
        bool active[C];
        int tcell[C];
        const VT *fp[C];  // the lane's cells as offsets from the corner (cells outside the region: the corner)
#pragma unroll
        for (int k = 0; k < C; ++k) {
            active[k] = ac + la < P.ea1 && bc + lb + k * hb < P.eb1;
            const int a = active[k] ? la : 0, b = active[k] ? lb + k * hb : 0;
            tcell[k] = (pw * nkR + pb * P.tile_b + b) * njR + pa * P.tile_a + a;
            const long long o = (long long)f * P.pstride + b * P.pna + a;
            if constexpr (MODE == MODE_GREY) fp[k] = P.fieldVG + o;
            else fp[k] = P.fieldVX + o;
        }
        const unsigned corner = ((unsigned)w0 * P.pnb + bc) * P.pna + ac;
        const int N = P.rays_per_packet ? P.rays_per_packet[G * P.rays_gstride + p] : P.rays;
        const float oW = (__ldg(P.fw + w0) + __ldg(P.fw + w0 + 1)) * 0.5f;
        // alias table of this packet: band group G of the temperature bin
        // nearest to the temperature of the packet's first cell
        int gs = 0, K = 1;
        if constexpr (MODE == MODE_GREY) {
            // T^4 with the sign set where the temperature is not positive
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const float v = __ldg(fp[k] + corner).x;
                if (active[k] && (__float_as_int(v) < 0 || v != v)) flags |= DNSMC_STATUS_BAD_FIELD;
            }
        } else {
            int boff = 0;
            if (P.n_tbins > 1) {
                const int4 v = __ldg(fp[0] + corner);
                const float tp0 = __shfl_sync(FULL, (float)(v.x >> 16) + __int_as_float(v.y), 0);
                int bin = __float2int_rn(tp0);
                bin = min(max(bin, 0), P.n_tbins - 1);
                boff = bin * P.n_groups;
            }
            gs = P.group_start[boff + G];
            K = P.group_start[boff + G + 1] - gs;
        }
        const uint32_t ctr2 = (uint32_t)G | ((uint32_t)(f + P.field_base) << 16);
        double mo[C][9];
        if (MOM)
#pragma unroll
            for (int k = 0; k < C; ++k)
#pragma unroll
                for (int q = 0; q < 9; ++q) mo[k][q] = 0.0;
        const int M = P.sampler ? max(1, N / max(1, P.nbatch)) : 1;
        if (!SPLIT)
#pragma unroll
        for (int k = 0; k < C; ++k) {
            *acc(0, k) = make_float2(0.0f, 0.0f); *acc(1, k) = make_float2(0.0f, 0.0f); *acc(2, k) = make_float2(0.0f, 0.0f);
        }
        unsigned long long isteps = 0;
        unsigned int lsteps = 0;  // this lane's active cell-steps in the item
        int rbeg = TRACE ? P.trace_r : 0;
        int rend = TRACE ? P.trace_r + 1 : ((K > 0) ? N : 0);
        float *const rayx = SPLIT ? P.rayx + item * N * 64 + lane : nullptr;
        if (SPLIT) unit_rays(P, part, rend, &rbeg, &rend);
        int m = P.sampler ? rbeg % M : 0;  // the ray's index in its replicate
        for (int r = rbeg; r < rend; ++r) {
            const int rb = (r - rbeg) & 31;
            if (rb == 0) {
                __syncwarp();
                if (r + lane < rend) ray_batch<MODE, TRACE, CV, true>(P, batch, r + lane, M, p, ctr2, gs, K, f, w0, lane);
                __syncwarp();
            }
            // the ray's table slab is on its way while the walk's first chunk
            // is generated
            float sW, sA, sB;
            int nbnd;
            {
                const float4 bw = batch->walk[rb], br = batch->rates[rb];
                sW = bw.x; sA = bw.y; sB = bw.z;
                nbnd = __float_as_int(br.z);
                if constexpr (MODE != MODE_GREY) slab_issue(P, __float_as_int(br.w), slab, lane, sbar);
            }
            float pab = 0.0f, psc = 0.0f;  // particle absorption / scattering per unit volume fraction
            if (P.part) { const float2 pp = __ldg(P.part + nbnd); pab = pp.x; psc = pp.y; }
            // the walk from (w.oW, fa0, fb0): the wall-normal coordinate and
            // the fractional offsets inside the current periodic cells (the
            // cell centres at emission, restarted at every scattering and wall
            // reflection)
            Walk w;
            float fa0 = 0.5f, fb0 = 0.5f;
            w.oW = oW;
            w.cw = w0; w.ca = ac; w.cb = bc;
            auto restart = [&]() {
                walk_direction(P, w, sW, sA, sB);
                // (an axis the ray does not move along is never crossed,
                // wherever the ray is in its cell)
                w.offA = w.dtA < INF ? (w.dA > 0 ? 1.0f - fa0 : fa0) : 0.5f;
                w.offB = w.dtB < INF ? (w.dB > 0 ? 1.0f - fb0 : fb0) : 0.5f;
            };
            restart();
            VT va[C], vb[C], vc[C], vd[C];  // field values of two steps and of the two after
#pragma unroll
            for (int k = 0; k < C; ++k) va[k] = __ldg(fp[k] + corner);
            float wk[C], Ii[C], tau[C], D[C];
            int life[C];  // steps each cell was live for (while it is: 2^30)
#pragma unroll
            for (int k = 0; k < C; ++k) {
                tau[k] = active[k] ? 1.0f : 0.0f;
                D[k] = 0.0f;
                life[k] = active[k] ? 1 << 30 : 0;
            }
            int steps = 0;
            // scattering events: one Philox word quadruple per event, a batch of
            // kEvents set up a lane each: free path, decision, azimuth; angle of
            // a scattering and of a reflection
            const float sigbar = P.fv_max * psc;
            uint32_t ev = 0;
            float4 e0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 *e1 = events;
            auto draw = [&]() {
                const uint32_t q = ev % kEvents;
                if (q == 0) {
                    __syncwarp();
                    if (lane < kEvents) {
                        const uint4 x = philox4x32_10(make_uint4((uint32_t)r, (uint32_t)p, ctr2, 0x5CA70000u + ev + lane), P.key0, P.key1);
                        float cp, sp, ct, st;
                        mc_sincos_turn(x.w >> 8, &cp, &sp);
                        hg_angle(P.hg_g, x.z, &ct, &st);
                        const float cmu = sqrtf(u24(x.z));
                        events[2 * lane] = make_float4(sigbar > 0.0f ? mc_neglog(u24o(x.x)) / sigbar : INF, u24(x.y), cp, sp);
                        events[2 * lane + 1] = make_float4(ct, st, cmu, sqrtf(fmaxf(0.0f, 1.0f - cmu * cmu)));
                    }
                    __syncwarp();
                }
                e0 = events[2 * q];
                e1 = events + 2 * q + 1;
                ++ev;
            };
            float tcol = INF;
            if (sigbar > 0.0f) { draw(); tcol = e0.x; }
            // One step of both cells, the same paired update as the gas
            // march's: e = expm1(k * (t - tn)) = -alpha, nta = tau e = -ta,
            // D += nta (-g), tau += nta; a cell already dumped (tau 0) adds
            // exactly nothing.
            auto step = [&](const VT (&v)[C], float nds, int s) {
                float kj[C], ngj[C];
#pragma unroll
                for (int h = 0; h < C; ++h) {
                    float fv;
                    if constexpr (MODE == MODE_GREY) {
                        ngj[h] = v[h].x - Ii[h];
                        kj[h] = P.kappa;
                        fv = v[h].y;
                    } else {
                        const float ft = __int_as_float(v[h].y);
                        kj[h] = lookup_k<MODE>(slk, v[h].x & 0xffff, ft, __int_as_float(v[h].z));
                        ngj[h] = lookup_ib(sli, v[h].x >> 16, ft) - Ii[h];
                        fv = __int_as_float(v[h].w);
                    }
                    kj[h] = fmaf(fv, pab, kj[h]);
                }
                const float2 e = mc_expm1_x2(__fmul2_rn(make_float2(kj[0], kj[1]), make_float2(nds, nds)));
                const float2 nta = __fmul2_rn(make_float2(tau[0], tau[1]), e);
                const float2 d2 = __ffma2_rn(nta, make_float2(ngj[0], ngj[1]), make_float2(D[0], D[1]));
                const float2 t2 = __fadd2_rn(make_float2(tau[0], tau[1]), nta);
                D[0] = d2.x; D[1] = d2.y;
                tau[0] = t2.x; tau[1] = t2.y;
#pragma unroll
                for (int h = 0; h < C; ++h) {
                    if (tau[h] < P.toll) {
                        D[h] = fmaf(-tau[h], ngj[h], D[h]);
                        tau[h] = 0.0f;
                        life[h] = min(life[h], s + 1);
                    }
                }
                if (TRACE && lane == 0 && s < P.trace_max) P.trace_rec[6 * s + 5] = __float_as_int(tau[0]);
            };
            bool first = true;
            for (;;) {  // chunks of the walk
                int end;
                const int n = walk_chunk<TRACE, true, 32>(P, w, (float)(walk_cap(false) - 4), min(walk_cap(false), P.max_steps - steps), tcol,
                                                      wbuf, lane, &end, steps);
                {
                    const unsigned c1 = n ? __float_as_uint(wbuf[3]) : corner;
#pragma unroll
                    for (int k = 0; k < C; ++k) vb[k] = __ldg(fp[k] + c1);
                }
                if (first) {
                    first = false;
                    if constexpr (MODE != MODE_GREY)
                        if (!slab_wait(P, sbar, &sphase, &flags)) { dead = true; break; }
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        if constexpr (MODE == MODE_GREY) {
                            Ii[k] = va[k].x;
                            wk[k] = P.W4sig * fmaf(va[k].y, pab, P.kappa);
                        } else {
                            const float ft = __int_as_float(va[k].y);
                            float ki = lookup_k<MODE>(slk, va[k].x & 0xffff, ft, __int_as_float(va[k].z));
                            ki = fmaf(__int_as_float(va[k].w), pab, ki);
                            Ii[k] = lookup_ib(sli, va[k].x >> 16, ft);
                            wk[k] = batch->walk[rb].w * ki;
                        }
                    }
                }
                bool done = false;
                if (n) {
                    // two steps on v0, v1 while the two after are fetched into
                    // v2, v3; the exit vote after the second
                    const float4 *wp = reinterpret_cast<const float4 *>(wbuf + 4);
                    float4 wc = wp[0];
                    int s = 0;
                    auto pair = [&](const VT (&v0)[C], const VT (&v1)[C], VT (&v2)[C], VT (&v3)[C]) {
                        const unsigned o2 = __float_as_uint(wc.y), o3 = __float_as_uint(wc.w);
#pragma unroll
                        for (int k = 0; k < C; ++k) v2[k] = __ldg(fp[k] + o2);
#pragma unroll
                        for (int k = 0; k < C; ++k) v3[k] = __ldg(fp[k] + o3);
                        const float d0 = wc.x, d1 = wc.z;
                        wc = *++wp;
                        step(v0, d0, steps + s);
                        step(v1, d1, steps + s + 1);
                        done = !__any_sync(FULL, tau[0] > 0.0f || tau[1] > 0.0f);
                        s += 2;
                    };
                    for (;;) {
                        pair(va, vb, vc, vd);
                        if (done || s >= n) break;
                        pair(vc, vd, va, vb);
                        if (done || s >= n) break;
                    }
                    steps += n;
                    walk_state<32>(wbuf, w);
                }
                if (done) break;  // every cell dumped
                if (end == WALK_WALL) {
                    const int side = w.dW > 0 ? 1 : 0;
                    const float Iw = (MODE == MODE_GREY) ? P.Tw4[side] : __ldg(P.ibw + side * P.nbands + nbnd);
                    // grey wall: it takes eps of the throughput at its
                    // own intensity and reflects the rest diffusely
                    const float eps = P.eps[side];
                    bool live = false;
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        if (tau[k] > 0.0f) {
                            const float gw = Ii[k] - Iw;
                            D[k] = fmaf(tau[k] * eps, gw, D[k]);
                            tau[k] = eps >= 1.0f ? 0.0f : tau[k] * (1.0f - eps);
                            if (tau[k] > 0.0f && tau[k] < P.toll) { D[k] = fmaf(tau[k], gw, D[k]); tau[k] = 0.0f; }
                            if (!(tau[k] > 0.0f)) life[k] = min(life[k], steps);
                        }
                        live = live || tau[k] > 0.0f;
                    }
                    if (!__any_sync(FULL, live)) break;
                    // diffuse reflection from the wall point
                    const float ta_ = w.t / w.dtA, tb_ = w.t / w.dtB;
                    fa0 = w.dA > 0 ? fa0 + (ta_ - w.nA) : fa0 - (ta_ - w.nA);
                    fb0 = w.dB > 0 ? fb0 + (tb_ - w.nB) : fb0 - (tb_ - w.nB);
                    fa0 = fminf(fmaxf(fa0, 0.0f), 1.0f);
                    fb0 = fminf(fmaxf(fb0, 0.0f), 1.0f);
                    w.oW = side == 0 ? __ldg(P.fw) : __ldg(P.fw + P.nw);
                    draw();  // this event's words: the reflected direction only
                    const float4 e = *e1;
                    sW = side == 0 ? e.z : -e.z;
                    sA = e.w * e0.z;
                    sB = e.w * e0.w;
                    restart();
                    if (sigbar > 0.0f) { draw(); tcol = e0.x; }
                    if (steps >= P.max_steps) {
                        if (live) flags |= DNSMC_STATUS_STEP_CAP;
                        break;
                    }
                } else if (steps >= P.max_steps || (n == 0 && end != WALK_COL)) {
                    // the step cap, or no walk through these faces
                    if (tau[0] > 0.0f || tau[1] > 0.0f) flags |= DNSMC_STATUS_STEP_CAP;
                    break;
                }
                // the cell the walk is in now
                const unsigned c0 = ((unsigned)w.cw * P.pnb + w.cb) * P.pna + w.ca;
#pragma unroll
                for (int k = 0; k < C; ++k) va[k] = __ldg(fp[k] + c0);
                if (end == WALK_COL) {
                    // tentative collision: a step to it, then the shared
                    // decision with per-cell weights
                    if (TRACE && lane == 0 && steps < P.trace_max) {
                        int *rec = P.trace_rec + 6 * steps;
                        rec[0] = w.cw; rec[1] = w.dA * (int)w.nA; rec[2] = w.dB * (int)w.nB; rec[3] = 3;
                        rec[4] = __float_as_int(tcol - w.t);
                    }
                    step(va, w.t - tcol, steps);
                    w.t = tcol;
                    ++steps;
                    float pl[C];
                    float ps = 0.0f, pc = 0.0f;
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const float fv = gen_fraction(va[k]);
                        pl[k] = tau[k] > 0.0f ? fminf(1.0f, fv * psc / sigbar) : 0.0f;
                        ps = k == 0 ? pl[k] : ps + pl[k];
                        pc = k == 0 ? (tau[k] > 0.0f ? 1.0f : 0.0f) : pc + (tau[k] > 0.0f ? 1.0f : 0.0f);
                    }
                    for (int o = 16; o > 0; o >>= 1) {
                        ps += __shfl_xor_sync(FULL, ps, o);
                        pc += __shfl_xor_sync(FULL, pc, o);
                    }
                    const float q = pc > 0.0f ? ps / pc : 0.0f;
                    const bool scatter = e0.y < q;
#pragma unroll
                    for (int k = 0; k < C; ++k)
                        if (tau[k] > 0.0f) {
                            tau[k] = tau[k] * (scatter ? pl[k] / q : (1.0f - pl[k]) / (1.0f - q));
                            if (!(tau[k] > 0.0f)) life[k] = min(life[k], steps);
                        }
                    float t0 = w.t;  // the next collision's time counts from here
                    if (scatter) {
                        const float ta_ = w.t / w.dtA, tb_ = w.t / w.dtB;
                        fa0 = w.dA > 0 ? fa0 + (ta_ - w.nA) : fa0 - (ta_ - w.nA);
                        fb0 = w.dB > 0 ? fb0 + (tb_ - w.nB) : fb0 - (tb_ - w.nB);
                        fa0 = fminf(fmaxf(fa0, 0.0f), 1.0f);
                        fb0 = fminf(fmaxf(fb0, 0.0f), 1.0f);
                        w.oW = fminf(fmaxf(fmaf(sW, w.t, w.oW), __ldg(P.fw + w.cw)), __ldg(P.fw + w.cw + 1));
                        const float4 e = *e1;
                        hg_turn(e.x, e.y, e0.z, e0.w, &sW, &sA, &sB);
                        restart();
                        t0 = 0.0f;
                    }
                    draw();
                    tcol = t0 + e0.x;
                    if (!__any_sync(FULL, tau[0] > 0.0f || tau[1] > 0.0f)) break;
                    if (steps >= P.max_steps) {
                        if (tau[0] > 0.0f || tau[1] > 0.0f) flags |= DNSMC_STATUS_STEP_CAP;
                        break;
                    }
                }
            }
            if (dead) break;
            // the walk's length: the steps of the cell that lived longest
            steps = min(steps, __reduce_max_sync(FULL, max(life[0], life[1])));
            if (TRACE && lane == 0) *P.trace_n = steps;
#pragma unroll
            for (int k = 0; k < C; ++k) lsteps += active[k] ? (unsigned)min(life[k], steps) : 0u;
            isteps += (unsigned long long)steps;
            const float4 sur = CV ? batch->sur[rb] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < C; ++k) {
                float X = wk[k] * D[k];
                if (CV) {
                    // Y_a: the ray through the layer-mean medium; Y_b: its own-layer part
                    const float Ya = wk[k] * (Ii[k] - sur.x);
                    const float Yb = wk[k] * (sur.y * (Ii[k] - sur.z));
                    if (MOM && active[k]) {
                        const double xd = X, ya = Ya, yb = Yb;
                        mo[k][0] += xd; mo[k][1] += ya; mo[k][2] += yb;
                        mo[k][3] = fma(xd, xd, mo[k][3]); mo[k][4] = fma(ya, ya, mo[k][4]);
                        mo[k][5] = fma(yb, yb, mo[k][5]); mo[k][6] = fma(xd, ya, mo[k][6]);
                        mo[k][7] = fma(xd, yb, mo[k][7]); mo[k][8] = fma(ya, yb, mo[k][8]);
                    }
                    const float2 beta = P.beta ? P.beta[fg * P.region_cells + tcell[k]] : make_float2(1.0f, -1.0f);
                    X = X - beta.x * Ya;  // tallied: X - beta_a Y_a - beta_b Y_b; the
                    X = X - beta.y * Yb;  // means beta . E[Y] are added back at finalize
                }
                if (active[k]) {
                    ++my_rays;
                    if (!isfinite(X)) flags |= DNSMC_STATUS_NONFINITE;
                    if (SPLIT) rayx[(long long)r * 64 + 32 * k] = X;
                    else tally_ray(P, X, m, M, acc(0, k), acc(1, k), acc(2, k));
                }
            }
            m = P.sampler && m == M - 1 ? 0 : m + 1;
        }
        if (dead) break;  // the item's sums are incomplete; the solve fails
        my_steps += lsteps;
        if (TRACE) return;
        if (SPLIT) {
            if (P.item_steps && lane == 0) atomicAdd(P.item_steps + item, isteps);
            if (unit_done(P, item, lane)) {
#pragma unroll
                for (int k = 0; k < C; ++k)
                    if (active[k]) P.tally[fg * P.region_cells + tcell[k]] = sum_rays<64>(P, rayx + 32 * k, K > 0 ? N : 0, M);
            }
            continue;
        }
        if (P.item_steps && lane == 0) P.item_steps[item] = isteps;
#pragma unroll
        for (int k = 0; k < C; ++k) {
            if (!active[k]) continue;
            const long long o = fg * P.region_cells + tcell[k];
            P.tally[o] = make_double2(ff_value(*acc(0, k)), ff_value(*acc(1, k)));
            if (MOM) {
                double *out = P.moments + o * 9;
#pragma unroll
                for (int q = 0; q < 9; ++q) out[q] = mo[k][q];
            }
        }
    }
    if (dead) slab_drain(sbar, sphase);
    // per-warp counters and status
    for (int o = 16; o > 0; o >>= 1) {
        my_rays += __shfl_xor_sync(FULL, my_rays, o);
        my_steps += __shfl_xor_sync(FULL, my_steps, o);
        flags |= __shfl_xor_sync(FULL, flags, o);
    }
    if (lane == 0) {
        if (my_rays) atomicAdd(P.counters + 0, my_rays);
        if (my_steps) atomicAdd(P.counters + 1, my_steps);
        if (flags) atomicOr(P.status, flags);
    }
}

// The two-cell march of a medium: the absorbing gas (march_pair_kernel; UNI:
// of the same absorption coefficient everywhere) or the general medium
// (march_gen_kernel).
template <int MODE, bool UNI, bool TRACE, bool CV, bool MOM, bool SPLIT, bool GEN> struct march_cells_kernel {
    static constexpr void (*fn)(const MarchParams) = march_pair_kernel<MODE, UNI, TRACE, CV, MOM, SPLIT>;
};
template <int MODE, bool UNI, bool TRACE, bool CV, bool MOM, bool SPLIT> struct march_cells_kernel<MODE, UNI, TRACE, CV, MOM, SPLIT, true> {
    static constexpr void (*fn)(const MarchParams) = march_gen_kernel<MODE, TRACE, CV, MOM, SPLIT>;
};

template <bool GEN>
int launch_march_cells(int mode, const MarchParams &p, int blocks, int threads, void *stream, bool trace, bool cv,
                       bool mom) {
    cudaStream_t st = (cudaStream_t)stream;
    if (trace) { blocks = 1; threads = 32; mom = false; }
    const size_t smem = march_pair_smem(p, threads);
#define DNSMC_L(M, U, T, CV_, O, S) \
    return march_launch_one(march_cells_kernel<M, U, T, CV_, O, S, GEN>::fn, blocks, threads, smem, st, p)
#define DNSMC_MODE(M, U)                                                                                \
    if (trace) { if (cv) DNSMC_L(M, U, true, true, false, false); else DNSMC_L(M, U, true, false, false, false); } \
    else if (cv && mom) DNSMC_L(M, U, false, true, true, false);                                        \
    else if (p.parts > 1) {                                                                             \
        if (cv) DNSMC_L(M, U, false, true, false, true); else DNSMC_L(M, U, false, false, false, true); \
    } else if (cv) DNSMC_L(M, U, false, true, false, false);                                            \
    else DNSMC_L(M, U, false, false, false, false);
    switch (mode) {
        case MODE_GREY: DNSMC_MODE(MODE_GREY, !GEN) break;
        case MODE_T:
            if constexpr (!GEN) {
                if (p.uni) { DNSMC_MODE(MODE_T, true) break; }
            }
            DNSMC_MODE(MODE_T, false) break;
        case MODE_TX: DNSMC_MODE(MODE_TX, false) break;
        default: break;
    }
#undef DNSMC_MODE
#undef DNSMC_L
    return (int)cudaErrorInvalidValue;
}

template <bool GEN>
int march_cells_occupancy(int mode, bool uni, int threads, bool cv, bool mom, size_t smem) {
    int nb = 0;
#define DNSMC_O(M, U)                                                                                     \
    nb = cv ? (mom ? march_occupancy_one(march_cells_kernel<M, U, false, true, true, false, GEN>::fn, threads, smem)     \
                   : march_occupancy_one(march_cells_kernel<M, U, false, true, false, false, GEN>::fn, threads, smem))   \
            : march_occupancy_one(march_cells_kernel<M, U, false, false, false, false, GEN>::fn, threads, smem)
    if (mode == MODE_GREY) DNSMC_O(MODE_GREY, !GEN);
    if (mode == MODE_T) {
        if (!GEN && uni) DNSMC_O(MODE_T, !GEN);
        else DNSMC_O(MODE_T, false);
    }
    if (mode == MODE_TX) DNSMC_O(MODE_TX, false);
#undef DNSMC_O
    return nb > 0 ? nb : 1;
}

}  // namespace dnsmc
