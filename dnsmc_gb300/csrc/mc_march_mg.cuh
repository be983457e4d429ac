// mc_march_mg.cuh -- the multigrid march (grid_num > 1; the reference's grid
// switch, code/mc_gpu.cu:193-207), one cell per lane, 32-cell packets: the
// absorbing gas with black walls, grey or T tables, no control variate.
// Instantiated in mc_kernels.cu.
#pragma once
#include "mc_march_pair.cuh"

namespace dnsmc {

// Persistent: every warp pulls work items (field, band group, packet), or
// units of an item's rays (SPLIT), from an atomic counter.  The fine phase is
// a warp-uniform walk for mg_steps steps; then every lane continues from its
// own point on the coarser grids with the reference's position-update march.
//
// It is bound by issue (the coarse steps, each lane with its own faces), so a
// step keeps what it can between steps: cell and face indices advanced, the
// periodic axes mirrored so that rays run up, table coordinates per coarse
// cell instead of its temperature, the next cell chosen by predicates instead
// of branches, and what a level's steps share held in registers (keep: the
// compiler otherwise computes most of it again in every step).  UNI: the
// absorption coefficient is the same everywhere (grey model, grey band
// tables).  The rays are set up a lane each, 32 at a time.  Instructions a
// coarse step 108 (163 without all this); 64^3, five levels, 60 rays: 1.37 ms
// (1.93).
//
// A value the compiler keeps instead of computing it again in every step.
__device__ __forceinline__ float keep(float v) { asm volatile("" : "+f"(v)); return v; }
template <class T>
__device__ __forceinline__ T *keep(T *v) { asm volatile("" : "+l"(v)); return v; }
__device__ __forceinline__ int keep(int v) { asm volatile("" : "+r"(v)); return v; }

// lookup_ib at a shared-memory address
__device__ __forceinline__ float lookup_ib_at(int ibs, int ti, float ft) {
    float a, d;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a), "=f"(d) : "r"(ibs + ti * 8));
    return fmaf(ft, d, a);
}

// Resident blocks of 256 threads per SM the register allocation must allow
// (2: up to 128 registers; 3: 85; 4: 64): the march takes 1.47 / 1.48 / 1.48 ms
// (before the rays were set up together).
#ifndef DNSMC_MINB
#define DNSMC_MINB 4
#endif
template <int MODE, bool UNI, bool TRACE, bool SPLIT>
__global__ void __launch_bounds__(256, DNSMC_MINB) march_mg_kernel(const MarchParams P) {
    typedef typename FieldT<MODE>::type VT;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int la = lane % P.tile_a, lb = lane / P.tile_a;
    const int njR = P.ea1 - P.ea0, nkR = P.eb1 - P.eb0;
    unsigned long long my_rays = 0, my_steps = 0;
    unsigned int flags = 0;
    const int tid = threadIdx.x;
    // dynamic shared memory (march_mg_smem): this warp's copy of the current
    // ray's table slab (tabulated models), its ray batch, then the item's sums
    // as float pairs [3][threads]
    extern __shared__ float4 s_dyn[];
    const int nthr = blockDim.x;
    const int warp = threadIdx.x >> 5, nwarp = (nthr + 31) >> 5;
    float2 *const slk = reinterpret_cast<float2 *>(s_dyn) + warp * P.slab_len;
    const float2 *const sli = slk + P.slab_klen;
    unsigned char *const s_batch = reinterpret_cast<unsigned char *>(reinterpret_cast<float2 *>(s_dyn) + nwarp * P.slab_len);
    RayBatch *const batch = reinterpret_cast<RayBatch *>(s_batch + warp * kMgBatchBytes);  // walk and rates only
    float2 *const s_acc = reinterpret_cast<float2 *>(s_batch + nwarp * kMgBatchBytes);
    // each warp's transaction barrier of its slab copies, and its parity
    __shared__ uint64_t s_bar[8];
    uint64_t *const sbar = &s_bar[warp];
    uint32_t sphase = 0;
    slab_bar_init(sbar, lane);
    const int ibs = keep((int)smem_addr(sli));
    const float fna = keep((float)P.na), fnb = keep((float)P.nb);
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
        const int a0 = P.ea0 + pa * P.tile_a + la;
        const int b0 = P.eb0 + pb * P.tile_b + lb;
        const bool active = (a0 < P.ea1) && (b0 < P.eb1);
        const int acl = active ? a0 : P.ea0, bcl = active ? b0 : P.eb0;
        const int N = P.rays_per_packet ? P.rays_per_packet[G * P.rays_gstride + p] : P.rays;
        const long long fbase = (long long)f * P.field_stride;
        // own-cell quantities
        const VT *field;
        if constexpr (MODE == MODE_T) field = P.fieldP + fbase; else field = P.fieldT + fbase;
        const int cell0 = (w0 * P.nb + bcl) * P.na + acl;
        const VT vown = __ldg(field + cell0);
        float Ti4 = 0.f, tpos0 = 0.f;
        int ti_i = 0, ki_i = 0;
        float ft_i = 0.f, fx_i = 0.f;
        if constexpr (MODE == MODE_GREY) {
            const float Ti = vown;
            if (!(Ti > 0.0f) && active) flags |= DNSMC_STATUS_BAD_FIELD;
            const float t2 = Ti * Ti;
            Ti4 = t2 * t2;
        } else {
            cell_coords<MODE>(vown, &ki_i, &ti_i, &ft_i, &fx_i);
            tpos0 = (float)ti_i + ft_i;  // the clamped table coordinate, exactly
        }
        const float oW = (__ldg(P.fw + w0) + __ldg(P.fw + w0 + 1)) * 0.5f;
        // alias table of this packet: band group G of the temperature bin
        // nearest to lane 0's temperature (one bin when sampling at Tmax)
        int gs = 0, K = 1;
        if (MODE != MODE_GREY) {
            int boff = 0;
            if (P.n_tbins > 1) {
                const float tp0 = __shfl_sync(FULL, tpos0, 0);
                int bin = __float2int_rn(tp0);
                bin = min(max(bin, 0), P.n_tbins - 1);
                boff = bin * P.n_groups;
            }
            gs = P.group_start[boff + G];
            K = P.group_start[boff + G + 1] - gs;
        }
        const uint32_t ctr2 = (uint32_t)G | ((uint32_t)(f + P.field_base) << 16);
        const long long tc = ((long long)(w0 - P.ew0) * nkR + (bcl - P.eb0)) * njR + (acl - P.ea0);
        const long long cell_out = fg * P.region_cells + tc;  // tally index of this lane's cell
        const int M = P.sampler ? max(1, N / max(1, P.nbatch)) : 1;
        if (!SPLIT) {
            s_acc[tid] = make_float2(0.0f, 0.0f); s_acc[nthr + tid] = make_float2(0.0f, 0.0f);
            s_acc[2 * nthr + tid] = make_float2(0.0f, 0.0f);
        }
        unsigned long long isteps = 0;
        unsigned int lsteps = 0;  // this lane's active steps in the item
        int rbeg = TRACE ? P.trace_r : 0;
        int rend = TRACE ? P.trace_r + 1 : ((K > 0) ? N : 0);
        float *const rayx = SPLIT ? P.rayx + item * N * 32 + lane : nullptr;
        if (SPLIT) unit_rays(P, part, rend, &rbeg, &rend);
        int m = P.sampler ? rbeg % M : 0;  // the ray's index in its replicate
        for (int r = rbeg; r < rend; ++r) {
            const int rb = (r - rbeg) & 31;
            if (rb == 0) {
                __syncwarp();
                if (r + lane < rend) {
                    ray_batch<MODE, TRACE, false, true>(P, batch, r + lane, M, p, ctr2, gs, K, f, w0, lane);
                    const float4 d = batch->walk[lane];
                    batch->rates[lane].x = 1.0f / fabsf(d.y);
                    batch->rates[lane].y = 1.0f / fabsf(d.z);
                }
                __syncwarp();
            }
            const float4 bw = batch->walk[rb], br = batch->rates[rb];
            if constexpr (MODE != MODE_GREY) slab_issue(P, __float_as_int(br.w), smem_addr(slk), lane, sbar);
            const float sW = bw.x, sA = bw.y, sB = bw.z;
            const int nbnd = __float_as_int(br.z);

            // fine phase: the warp-uniform DDA from the cell centres
            const float invW = 1.0f / fabsf(sW), invA = br.x, invB = br.y;
            const int dW = sW > 0.f ? 1 : -1, dA = sA > 0.f ? 1 : -1, dB = sB > 0.f ? 1 : -1;
            const float sinvW = dW > 0 ? invW : -invW;
            const float dtA = P.da * invA, dtB = P.db * invB;
            const float *const fwd = keep(P.fw + (dW > 0 ? 1 : 0));  // the face ahead of a cell
            int cw = w0, cell = cell0;
            const int cW1 = keep(dW * P.na * P.nb), cB1 = keep(dB * P.na);
            const int cA = keep(-dA * P.na), cB = keep(-dB * P.na * P.nb);  // back by a period
            // crossings so far (exact in FP32), the one that leaves the period,
            // and the walk's parameter
            float nA = 0.0f, nB = 0.0f, t = 0.0f;
            float eA = (float)(dA > 0 ? P.na - acl : acl + 1), eB = (float)(dB > 0 ? P.nb - bcl : bcl + 1);
            float tW = (__ldg(fwd + cw) - oW) * sinvW, tA = 0.5f * dtA, tB = 0.5f * dtB;
            float tau = active ? 1.0f : 0.0f;
            float D = 0.0f;
            int steps = 0;
            // ray weight (the ray contributes wk D, D the net exchange in
            // intensity units) and the own cell's intensity
            float wk = bw.w, Ii = Ti4;
            if constexpr (MODE != MODE_GREY) {
                if (!slab_wait(P, sbar, &sphase, &flags)) { dead = true; break; }
                const float ki = UNI ? P.kappa : lookup_k<MODE>(slk, ki_i, ft_i, fx_i);
                Ii = lookup_ib(sli, ti_i, ft_i);
                wk = bw.w * ki;
            }
            // One segment of length ds: alpha = 1 - exp(-k ds), ta = tau alpha, D +=
            // ta g, tau -= ta; a lane that has ended (tau 0) keeps its sum.
            auto absorb = [&](float kj, float gj, float ds) {
                const bool live = tau > 0.0f;
                const float ta = tau * -mc_expm1(-(kj * ds));
                float d = fmaf(ta, gj, D);
                tau = tau - ta;
                const bool low = tau < P.toll;
                d = low ? fmaf(tau, gj, d) : d;
                tau = low ? 0.0f : tau;
                D = live ? d : D;
            };
            auto wall_hit = [&](int side) {
                const float Iw = (MODE == MODE_GREY) ? P.Tw4[side] : __ldg(P.ibw + side * P.nbands + nbnd);
                if (tau > 0.0f) D = fmaf(tau, Ii - Iw, D);
                tau = 0.0f;
            };
            VT vcur = vown;
            for (;;) {
                const bool hw = tW <= tA && tW <= tB, ha = !hw && tA <= tB, hb = !hw && !ha;
                const float tn = fminf(tW, fminf(tA, tB)), ds = tn - t;
                if (TRACE && lane == 0 && steps < P.trace_max) {
                    int *rec = P.trace_rec + 6 * steps;
                    rec[0] = cw; rec[1] = dA * (int)nA; rec[2] = dB * (int)nB; rec[3] = hw ? 0 : ha ? 1 : 2;
                    rec[4] = __float_as_int(ds);
                }
                // the next cell, and its field value fetched now
                cell += hw ? cW1 : (ha ? dA : cB1);
                if (hw) cw += dW;
                if (ha) nA += 1.0f;
                if (hb) nB += 1.0f;
                if (nA == eA) { cell += cA; eA += fna; }
                if (nB == eB) { cell += cB; eB += fnb; }
                const bool wall = (unsigned)cw >= (unsigned)P.nw;
                VT vnext = vcur;
                if (!wall) {
                    vnext = __ldg(field + cell);
                    tW = (__ldg(fwd + cw) - oW) * sinvW;
                }
                float kj = P.kappa, gj;
                if constexpr (MODE == MODE_GREY) {
                    const float t2 = vcur * vcur;
                    gj = Ti4 - t2 * t2;
                } else {
                    int kx, tj;
                    float ftj, fxj;
                    cell_coords<MODE>(vcur, &kx, &tj, &ftj, &fxj);
                    if (!UNI) kj = lookup_k<MODE>(slk, kx, ftj, fxj);
                    gj = Ii - lookup_ib_at(ibs, tj, ftj);
                }
                if (tau > 0.0f) ++lsteps;
                absorb(kj, gj, ds);
                if (TRACE && lane == 0 && steps < P.trace_max) P.trace_rec[6 * steps + 5] = __float_as_int(tau);
                t = tn;
                ++steps;
                if (wall) { wall_hit(cw < 0 ? 0 : 1); break; }
                tA = (nA + 0.5f) * dtA; tB = (nB + 0.5f) * dtB;
                vcur = vnext;
                if (!__any_sync(FULL, tau > 0.0f) || steps >= P.mg_steps) break;
            }
            // Coarse grids: every lane continues from its own point; lanes no
            // longer share their cell faces, but they step in lockstep and
            // leave a level together.
            if (__any_sync(FULL, tau > 0.0f)) {
                const float ua = t / dtA - nA, ub = t / dtB - nB;
                const int ca = dA > 0 ? (int)(nA - (eA - fna)) : (int)(eA - nA) - 1;
                const int cb = dB > 0 ? (int)(nB - (eB - fnb)) : (int)(eB - nB) - 1;
                const float fa = fminf(fmaxf(dA > 0 ? 0.5f + ua : 0.5f - ua, 0.0f), 1.0f);
                const float fb = fminf(fmaxf(dB > 0 ? 0.5f + ub : 0.5f - ub, 0.0f), 1.0f);
                float xp = fmaf(sW, t, oW);
                // y and z are mirrored where the ray runs down (a change of sign
                // is exact), so that it runs up along both
                const float pA = dA > 0 ? 1.0f : -1.0f, pB = dB > 0 ? 1.0f : -1.0f;
                float yp = pA * (((float)ca + fa) * P.da);
                float zp = pB * (((float)cb + fb) * P.db);
                int ic = cw, jc = ca, kc = cb;
                // distance to the face ahead: (face - x) / s, infinite where s is 0
                // (s <= 0: the face lies below, -inf times a negative number)
                const float isx = keep(sinvW), isy = keep(invA), isz = keep(invB);
                const float sy = keep(fabsf(sA)), sz = keep(fabsf(sB)), Ii_ = keep(Ii);
                for (int l = 1; l < P.mg_levels; ++l) {
                    ic >>= 1; jc >>= 1; kc >>= 1;
                    const int nwL = P.nw >> l, naL = P.na >> l, nbL = P.nb >> l;
                    const float *const fwL = keep(P.mgfw + P.mg_fwoff[l] + (dW > 0 ? 1 : 0));
                    const float daL = keep(P.mg_da[l]), dbL = keep(P.mg_db[l]);
                    const long long lev = P.mg_off[l] + (long long)f * nwL * naL * nbL;
                    const float *const gT = MODE == MODE_GREY ? keep(P.mgT + lev) : nullptr;
                    const int2 *const gP = MODE == MODE_GREY ? nullptr : keep(P.mgP + lev);
                    // the cell's index, and along the periodic axes the (mirrored) index of
                    // the face ahead, exact in FP32, its value past the last face, and
                    // the position after a wrap
                    int c = (ic * nbL + kc) * naL + jc;
                    float fj = (float)(dA > 0 ? jc + 1 : -jc), fk = (float)(dB > 0 ? kc + 1 : -kc);
                    const float fnj = keep((float)naL), fnk = keep((float)nbL);
                    const float ej = keep(dA > 0 ? fnj + 1.0f : 1.0f), ek = keep(dB > 0 ? fnk + 1.0f : 1.0f);
                    const float wy = keep(dA > 0 ? 0.0f : -P.Ly), wz = keep(dB > 0 ? 0.0f : -P.Lz);
                    const int sW1 = keep(dW * naL * nbL), sB1 = keep(dB * naL), rA = keep(-dA * naL), rB = keep(-dB * naL * nbL);
                    const int cap = (l == P.mg_levels - 1) ? P.max_steps : P.mg_steps;
                    int lv = 0;  // this lane's steps on the level
                    for (int counter = 0; counter < cap; ++counter) {
                        // the vote at every other step: lanes that have ended walk on
                        // (traced, they stand)
                        if ((TRACE || !(counter & 1)) && !__any_sync(FULL, tau > 0.0f)) break;
                        float dsr = 0.0f;  // this lane's segment (0 when it idles)
                        if (!TRACE || tau > 0.0f) {
                            const float fx = __ldg(fwL + ic);
                            const float fy = fj * daL, fz = fk * dbL;
                            const float dsx = (fx - xp) * isx, dsy = (fy - yp) * isy, dsz = (fz - zp) * isz;
                            float kj = P.kappa, gj;
                            if constexpr (MODE == MODE_GREY) {
                                const float Tc = __ldg(gT + c), t2 = Tc * Tc;
                                gj = Ii_ - t2 * t2;
                            } else {
                                const int2 v = __ldg(gP + c);
                                const float ftj = __int_as_float(v.y);
                                if (!UNI) kj = lookup_k<MODE_T>(slk, v.x, ftj, 0.0f);
                                gj = Ii_ - lookup_ib_at(ibs, v.x, ftj);
                            }
                            const float dmin = fminf(fminf(dsx, dsy), dsz);
                            const float ds = fmaxf(dmin, 0.0f);
                            if (TRACE) dsr = ds;
                            xp = dmin == dsx ? fx : fmaf(ds, sW, xp);
                            yp = dmin == dsy ? fy : fmaf(ds, sy, yp);
                            zp = dmin == dsz ? fz : fmaf(ds, sz, zp);
                            if (tau > 0.0f) ++lv;
                            absorb(kj, gj, ds);
                            const bool xy = dsx < dsy;
                            const bool hw = xy && dsx < dsz, ha = !xy && dsy < dsz;
                            c += hw ? sW1 : (ha ? dA : sB1);
                            if (hw) ic += dW;
                            if (ha) fj += 1.0f;
                            if (!hw && !ha) fk += 1.0f;
                            if (fj == ej) { fj -= fnj; yp = wy; c += rA; }
                            if (fk == ek) { fk -= fnk; zp = wz; c += rB; }
                            if ((unsigned)ic >= (unsigned)nwL) {
                                wall_hit(ic < 0 ? 0 : 1);
                                ic -= dW;
                                c -= sW1;
                            }
                        }
                        if (TRACE && lane == 0 && steps + counter < P.trace_max) {  // every iteration
                            int *rec = P.trace_rec + 6 * (steps + counter);
                            rec[0] = ic; rec[1] = dA > 0 ? (int)fj - 1 : -(int)fj; rec[2] = dB > 0 ? (int)fk - 1 : -(int)fk; rec[3] = 16 + l;
                            rec[4] = __float_as_int(dsr); rec[5] = __float_as_int(tau);
                        }
                    }
                    jc = dA > 0 ? (int)fj - 1 : -(int)fj;
                    kc = dB > 0 ? (int)fk - 1 : -(int)fk;
                    lsteps += lv;
                    steps += __reduce_max_sync(FULL, lv);  // until the last lane's end
                }
                if (tau > 0.0f) flags |= DNSMC_STATUS_STEP_CAP;
            }
            if (TRACE && lane == 0) *P.trace_n = steps;
            isteps += (unsigned long long)steps;
            const float X = wk * D;
            if (active) {
                ++my_rays;
                if (!isfinite(X)) flags |= DNSMC_STATUS_NONFINITE;
                if (SPLIT) rayx[(long long)r * 32] = X;
                else tally_ray(P, X, m, M, &s_acc[tid], &s_acc[nthr + tid], &s_acc[2 * nthr + tid]);
            }
            m = P.sampler && m == M - 1 ? 0 : m + 1;
        }
        if (dead) break;  // the item's sums are incomplete; the solve fails
        my_steps += lsteps;
        if (TRACE) return;
        if (SPLIT) {
            if (P.item_steps && lane == 0) atomicAdd(P.item_steps + item, isteps);
            if (unit_done(P, item, lane) && active) P.tally[cell_out] = sum_rays<32>(P, rayx, K > 0 ? N : 0, M);
            continue;
        }
        if (P.item_steps && lane == 0) P.item_steps[item] = isteps;
        if (active) P.tally[cell_out] = make_double2(ff_value(s_acc[tid]), ff_value(s_acc[nthr + tid]));
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

// The kernel of a launch: traces take the table lookups (the same results).
inline void (*march_mg_fn(int mode, bool uni, bool split, bool trace))(const MarchParams) {
    if (mode == MODE_GREY)
        return trace ? march_mg_kernel<MODE_GREY, true, true, false>
                     : split ? march_mg_kernel<MODE_GREY, true, false, true> : march_mg_kernel<MODE_GREY, true, false, false>;
    if (mode != MODE_T) return nullptr;
    if (trace) return march_mg_kernel<MODE_T, false, true, false>;
    if (uni) return split ? march_mg_kernel<MODE_T, true, false, true> : march_mg_kernel<MODE_T, true, false, false>;
    return split ? march_mg_kernel<MODE_T, false, false, true> : march_mg_kernel<MODE_T, false, false, false>;
}

}  // namespace dnsmc
