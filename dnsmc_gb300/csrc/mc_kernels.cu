// mc_kernels.cu -- sm_103a device code of the reverse (emission-based, OERM)
// Monte Carlo radiative-source solver.
//
// Replaces kernel_fluid / march_ray / find_band / emiss_ang / kernel_results
// of the reference (code/mc_gpu.cu:44-438, :813-896, :959-970) with persistent
// work-queue kernels built around "packets" (mc_march_pair.cuh on the fine grid,
// mc_march_mg.cuh with coarse grids): cells of one wall-normal plane that tile
// the periodic (j, k) plane and are owned by one warp.  Every ray of a packet
// shares one draw -- direction (reference emiss_ang, code/mc_gpu.cu:813-820) and
// spectral sample (find_band, :830-896) -- and with it the voxel walk, since the
// origins differ by whole periodic cells; the lanes do the OERM update of
// march_ray (:264-276) for their own cells.
//
// This file: what surrounds the marches -- packing and statistics of the fields,
// table coordinates and slabs, the control variate's preparation and means, the
// queue order, the ray counts by optical thickness, the multigrid march's
// launch and coarsening, the finalize.
//
// Rays are drawn either iid (one Philox4x32-10 call per packet-ray) or as
// randomised quasi-Monte Carlo: the N rays of a (packet, band group) are
// nbatch replicates of the first N/nbatch points of a 4-dimensional Sobol' net
// (phi, cos theta, spectral index, alias threshold), each replicate XOR-shifted
// by a Philox word; the spectral sample comes from the alias table of the
// packet's own temperature bin when local sampling is on.
//
// Arithmetic is FP32 with explicit fmaf and the file is compiled with
// -fmad=false, so the host replay reproduces every ray bit for bit; exp and
// sin/cos are the project's own polynomial kernels (mc_expm1 / mc_sincos) for
// the same reason.
#include <atomic>

#include "mc_march_mg.cuh"

namespace dnsmc {

// Table coordinates of the field for the march: p = clamp((T - T0)/dT, 0,
// nT-1) (and the same for x_H2O), computed once per solve with the same FP32
// operations the march used to apply per step; or T^4 for the grey model.
// Row by row of the output, a thread per j.
__global__ void field_pos_kernel(const FieldPos q) {
    const long long rows = (long long)q.nfields * q.nw * q.pnb, n = rows * q.pna;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / q.pna, fw = r / q.pnb;
        int a = (int)(i - r * q.pna), b = (int)(r - fw * q.pnb);
        a = a >= q.na ? a - q.na : a;
        b = b >= q.nb ? b - q.nb : b;
        const long long src = (fw * q.nb + b) * q.na + a;
        int ti, xi;
        float ft, fx;
        const float fv = q.fV ? q.fV[src] : 0.0f;
        if (q.outG || q.outVG) {
            const float T = q.fT[src], t2 = T * T, v = t2 * t2;
            if (q.outG) q.outG[i] = T > 0.0f ? v : -v;
            else q.outVG[i] = make_float2(T > 0.0f ? v : -v, fv);
        } else if (q.fTX) {
            const float2 v = q.fTX[src];
            float pt = (v.x - q.T0) * q.invdT;
            pt = fminf(fmaxf(pt, 0.0f), (float)(q.nT - 1));
            float px = (v.y - q.X0) * q.invdX;
            px = fminf(fmaxf(px, 0.0f), (float)(q.nX - 1));
            pos_split(pt, q.nT, &ti, &ft);
            pos_split(px, q.nX, &xi, &fx);
            const int kx = ti * (q.nX - 1) + xi;  // below 2^16, as ti: the march's slab fits shared memory
            if (q.outVX) q.outVX[i] = make_int4(kx | ti << 16, __float_as_int(ft), __float_as_int(fx), __float_as_int(fv));
            else q.outPX[i] = make_int4(kx, __float_as_int(ft), __float_as_int(fx), ti);
        } else {
            float pt = (q.fT[src] - q.T0) * q.invdT;
            pt = fminf(fmaxf(pt, 0.0f), (float)(q.nT - 1));
            if (q.outF) {
                q.outF[i] = pt;
                continue;
            }
            pos_split(pt, q.nT, &ti, &ft);
            if (q.outVX) q.outVX[i] = make_int4(ti | ti << 16, __float_as_int(ft), 0, __float_as_int(fv));
            else q.outP[i] = make_int2(ti, __float_as_int(ft));
        }
    }
}

// ---------------------------------------------------------------------------
// Finalize: per cell of the region, Q = sum over groups of the group means,
// var(Q) = sum of the variances of the group means (groups are independent
// strata).  Replaces kernel_results + the host scatter (code/mc_gpu.cu:959-970,
// :762-776); the output is dense, i fastest.
// ---------------------------------------------------------------------------
// One block per tile of 32 j x 32 i cells of a k row of a field: the tally
// layout has j fastest and the outputs i fastest, so the block reads its
// cells along j (thread x = j) and writes them along i through a
// shared-memory transpose.  Every cell's arithmetic is in the same order as
// a plain per-cell loop over the groups.
constexpr int kFinTile = 32, kFinRows = 8;
__global__ void __launch_bounds__(kFinTile * kFinRows) finalize_kernel(const FinalizeParams F) {
    __shared__ double s_a[kFinTile][kFinTile + 1], s_b[kFinTile][kFinTile + 1];  // [i][j]
    const int tx = threadIdx.x % kFinTile, ty = threadIdx.x / kFinTile;
    const int ntj = (F.njR + kFinTile - 1) / kFinTile;
    const int j0 = (blockIdx.x % ntj) * kFinTile, i0 = (blockIdx.x / ntj) * kFinTile;
    const int kR = blockIdx.y, f = blockIdx.z;
    constexpr int S = kFinTile / kFinRows;  // cells per thread
    // read side: cell s of this thread is (iR = i0 + ty + kFinRows s, jR = j0 + tx)
    const int jR = j0 + tx;
    double Q[S], V[S];
#pragma unroll
    for (int s = 0; s < S; ++s) { Q[s] = 0.0; V[s] = 0.0; }
    // write side: thread x = i, cell s at (iR = i0 + tx, jR = j0 + ty + kFinRows s)
    const int iW = i0 + tx;
    for (int g = 0; g < F.n_groups; ++g) {
        double mg[S], vg[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int iR = i0 + ty + kFinRows * s;
            double m = 0.0, v = 0.0;
            if (iR < F.niR && jR < F.njR) {
                const long long tc = ((long long)iR * F.nkR + kR) * F.njR + jR;
                const int p = (iR * F.npb + kR / F.tile_b) * F.npa + jR / F.tile_a;
                const int N = F.rays_per_packet ? F.rays_per_packet[g * F.rays_gstride + p] : F.rays;
                const long long ti = ((long long)f * F.n_groups + g) * F.region_cells + tc;
                if (!F.group_empty[g] && N > 0) {
                    // divisions by the ray counts as products with their
                    // reciprocals (FP64 division is a long sequence on this GPU)
                    const double2 r = F.rays_per_packet ? F.rcp[g * F.rays_gstride + p] : F.rcp_uniform;
                    const double2 t = F.tally[ti];
                    m = t.x * r.x;
                    if (F.batched) {
                        if (F.nbatch > 1) v = fmax(0.0, t.y * F.rcp_batch.x - m * m) * F.rcp_batch.y;
                    } else if (N > 1) {
                        v = fmax(0.0, t.y * r.x - m * m) * r.y;
                    }
                }
                if (F.muY && !F.group_empty[g]) {
                    const float2 b = F.beta ? F.beta[ti] : make_float2(1.0f, -1.0f);
                    const double2 mu = F.muY[ti];
                    // Q_g = beta_a E[Y_a] + beta_b E[Y_b] + mean(X - beta_a Y_a - beta_b Y_b)
                    m += (double)b.x * mu.x;
                    m += (double)b.y * mu.y;
                }
            }
            Q[s] += m;
            V[s] += v;
            mg[s] = m;
            vg[s] = v;
        }
        if (F.Qg) {  // the group's results, [f][group][cell] i fastest
#pragma unroll
            for (int s = 0; s < S; ++s) { s_a[ty + kFinRows * s][tx] = mg[s]; s_b[ty + kFinRows * s][tx] = vg[s]; }
            __syncthreads();
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int jW = j0 + ty + kFinRows * s;
                if (iW < F.niR && jW < F.njR) {
                    const long long o = ((long long)f * F.n_groups + g) * F.region_cells +
                                        ((long long)kR * F.njR + jW) * F.niR + iW;
                    F.Qg[o] = s_a[tx][ty + kFinRows * s];
                    F.varg[o] = s_b[tx][ty + kFinRows * s];
                }
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int s = 0; s < S; ++s) { s_a[ty + kFinRows * s][tx] = Q[s]; s_b[ty + kFinRows * s][tx] = V[s]; }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int jW = j0 + ty + kFinRows * s;
        if (iW < F.niR && jW < F.njR) {
            const double Qc = s_a[tx][ty + kFinRows * s], Vc = s_b[tx][ty + kFinRows * s];
            const long long idx = (long long)f * F.region_cells + ((long long)kR * F.njR + jW) * F.niR + iW;
            F.Q[idx] = Qc;
            F.var[idx] = Vc;
            const double sd = sqrt(Vc);
            if (F.sigma) F.sigma[idx] = sd;
            if (F.Qf) {  // the float results the host receives (8 bytes per cell)
                F.Qf[idx] = (float)Qc;
                // one FP64 square root per cell when no scale applies
                F.sigf[idx] = (float)(F.sig_scale == 1.0 ? sd : sqrt(Vc * F.sig_scale));
            }
        }
    }
}

// Transpose a host-order field (i fastest, optional ghost layer) into the
// device order [i][k][j].  One thread per destination cell.
__global__ void pack_T_kernel(const float *src, float *dst, int nw, int na, int nb,
                              long long si, long long sj, long long sk, long long base) {
    const long long n = (long long)nw * na * nb;
    for (long long d = blockIdx.x * (long long)blockDim.x + threadIdx.x; d < n;
         d += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(d % na);
        const long long r = d / na;
        const int b = (int)(r % nb);
        const int w = (int)(r / nb);
        dst[d] = src[base + w * si + a * sj + b * sk];
    }
}

__global__ void pack_T4_kernel(const float *src, float *dst, int nw, int na, int nb, int pna, int pnb) {
    const long long n = (long long)nw * pnb * pna;
    for (long long d = blockIdx.x * (long long)blockDim.x + threadIdx.x; d < n; d += (long long)gridDim.x * blockDim.x) {
        const long long r = d / pna;
        int a = (int)(d - r * pna), b = (int)(r % pnb);
        const int w = (int)(r / pnb);
        a = a >= na ? a - na : a;
        b = b >= nb ? b - nb : b;
        const float T = src[w + (long long)nw * (a + (long long)na * b)], t2 = T * T, v = t2 * t2;
        dst[d] = T > 0.0f ? v : -v;
    }
}

__global__ void pack_TX_kernel(const float *srcT, const float *srcX, float2 *dst, int nw, int na,
                               int nb, long long si, long long sj, long long sk, long long base) {
    const long long n = (long long)nw * na * nb;
    for (long long d = blockIdx.x * (long long)blockDim.x + threadIdx.x; d < n;
         d += (long long)gridDim.x * blockDim.x) {
        const int a = (int)(d % na);
        const long long r = d / na;
        const int b = (int)(r % nb);
        const int w = (int)(r / nb);
        const long long s = base + w * si + a * sj + b * sk;
        dst[d] = make_float2(srcT[s], srcX ? srcX[s] : 0.0f);
    }
}

// Table slabs (launch_slabs), a pair a thread.  On the host this was 60 us of
// each solve with grey band tables, which depend on the fields' Tmax (1000
// bands: 0.9 MB of pairs).
__global__ void slab_kernel(const float *k, const float *ib, float2 *slab, int nS, int nq, int nT, int nX, int klen, int len) {
    const long long n = (long long)nS * len;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long sid = i / len;
        const int e = (int)(i - sid * len);
        float a = 0.0f, b = 0.0f;
        if (e < klen) {
            const float *r = k + sid * nT * nX;
            if (nX > 1) {  // pairs 2 c, 2 c + 1 of table cell c: rows t and t + 1
                const int c = e >> 1, t = c / (nX - 1), x = c - t * (nX - 1);
                r += (t + (e & 1)) * nX + x;
            } else {
                r += e;
            }
            a = r[0]; b = r[1];
        } else if (e < klen + nT - 1) {
            const float *r = ib + (sid / nq) * nT + (e - klen);
            a = r[0]; b = r[1];
        } else if (e == klen + nT - 1) {  // the last cell's interpolant at its end
            const float *r = ib + (sid / nq) * nT + nT - 2;
            a = b = fmaf(1.0f, r[1] - r[0], r[0]);
        }
        slab[i] = make_float2(a, b - a);
    }
}

// Extremes, sum and count of refused values of n cells (launch_field_stats) in
// a fixed order (deterministic): a grid-strided
// share per block, then the block that finishes last reduces the blocks' parts
// as the threads' were: 9 us at 64^3 and 5 us at 8 x 32 x 4 (two launches, the
// second one thread reading 256 parts in turn: 71 us).
// out: the four results, then the count of finished blocks (zero between
// launches).
constexpr int kStatBlocks = 256, kStatThreads = 256;
static_assert(kStatBlocks == kStatThreads, "the last block takes a part a thread");
struct FieldStats { double mx, mn, sm, bad; };
__device__ __forceinline__ FieldStats stats_merge(const FieldStats &a, const FieldStats &b) {
    return {fmax(a.mx, b.mx), fmin(a.mn, b.mn), a.sm + b.sm, a.bad + b.bad};
}
__device__ __forceinline__ FieldStats stats_block(FieldStats v, FieldStats *s) {
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = kStatThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] = stats_merge(s[threadIdx.x], s[threadIdx.x + o]);
        __syncthreads();
    }
    return s[0];
}
// A block's part of the statistics; the block that finishes last merges them all.
__device__ __forceinline__ void stats_finish(const FieldStats &v, FieldStats *s, FieldStats *part, double *out) {
    __shared__ bool last;
    const FieldStats b = stats_block(v, s);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(reinterpret_cast<unsigned int *>(out + 4), 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double *p = reinterpret_cast<const double *>(part + threadIdx.x);
    __syncthreads();
    FieldStats q = {-INFINITY, INFINITY, 0.0, 0.0};
    if (threadIdx.x < gridDim.x) q = {__ldcg(p), __ldcg(p + 1), __ldcg(p + 2), __ldcg(p + 3)};
    const FieldStats t = stats_block(q, s);
    if (threadIdx.x == 0) {
        out[0] = t.mx; out[1] = t.mn; out[2] = t.sm; out[3] = t.bad;
        *reinterpret_cast<unsigned int *>(out + 4) = 0u;
    }
}

template <int KIND>
__global__ void __launch_bounds__(kStatThreads) field_stats_kernel(const float *v, long long n, FieldStats *part, double *out) {
    __shared__ FieldStats s[kStatThreads];
    // FP32 extremes and FP64 sums of this thread's share (few FP64
    // instructions: this GPU runs them at a small fraction of the FP32 rate)
    float mx = -INFINITY, mn = INFINITY;
    double sm = 0.0;
    int bad = 0;
    for (long long i = blockIdx.x * (long long)kStatThreads + threadIdx.x; i < n; i += (long long)gridDim.x * kStatThreads) {
        float T;
        if (KIND == STATS_TX) { const float2 tx = reinterpret_cast<const float2 *>(v)[i]; T = tx.x; sm += tx.y; } else { T = v[i]; }
        if (KIND == STATS_V) sm += T;
        if (!(KIND == STATS_V ? T >= 0.0f : T > 0.0f) || !isfinite(T)) ++bad;
        mx = fmaxf(mx, T); mn = fminf(mn, T);
    }
    stats_finish({(double)mx, (double)mn, sm, (double)bad}, s, part, out);
}

// A small field packed and its statistics taken in one launch.  set_fields from
// device arrays of T, two launches and one: 32^3 26.0 and 24.2 us, 64^3 26.4 and
// 23.9, 96^3 34.4 and 26.5, 128^3 38.8 and 36.7.  Fields beyond kPackStatsCells
// keep the packing's own grid: what a launch costs is under a hundredth of
// their solves.
template <bool TX>
__global__ void __launch_bounds__(kStatThreads) pack_stats_kernel(const float *srcT, const float *srcX, float *dst, unsigned na, unsigned nb,
                                                                 unsigned n, long long si, long long sj, long long sk, long long base,
                                                                 FieldStats *part, double *out) {
    __shared__ FieldStats s[kStatThreads];
    float mx = -INFINITY, mn = INFINITY;
    double sm = 0.0;
    int bad = 0;
    for (unsigned d = blockIdx.x * kStatThreads + threadIdx.x; d < n; d += gridDim.x * kStatThreads) {
        const unsigned r = d / na, a = d - r * na, w = r / nb, b = r - w * nb;
        const long long o = base + w * si + a * sj + b * sk;
        const float T = srcT[o];
        if (TX) {
            const float x = srcX[o];
            reinterpret_cast<float2 *>(dst)[d] = make_float2(T, x);
            sm += x;
        } else {
            dst[d] = T;
        }
        if (!(T > 0.0f) || !isfinite(T)) ++bad;
        mx = fmaxf(mx, T); mn = fminf(mn, T);
    }
    stats_finish({(double)mx, (double)mn, sm, (double)bad}, s, part, out);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static std::atomic<long long> g_launches{0};
void note_launch(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(std::memory_order_relaxed); }

static inline int grid_for(long long n, int threads) {
    long long b = (n + threads - 1) / threads;
    if (b > 4096) b = 4096;
    if (b < 1) b = 1;
    return (int)b;
}

int launch_march_ex(int mode, const MarchParams &p, int blocks, int threads, void *stream, bool trace, bool cv,
                    bool mom, bool gen) {
    if (gen) return launch_march_gen(mode, p, blocks, threads, stream, trace, cv, mom);
    return launch_march_pair(mode, p, blocks, threads, stream, trace, cv, mom);
}

int march_occupancy_ex(int mode, bool uni, int threads, bool cv, bool mom, bool gen, size_t smem) {
    if (gen) return march_gen_occupancy(mode, threads, cv, mom, smem);
    return march_pair_occupancy(mode, uni, threads, cv, mom, smem);
}

// Multigrid march (reference tables or grey model; no control variate, no
// particles, black walls).
int launch_march_mg(int mode, const MarchParams &p, int blocks, int threads, void *stream, bool trace) {
    cudaStream_t st = (cudaStream_t)stream;
    if (trace) { blocks = 1; threads = 32; }
    const auto k = march_mg_fn(mode, p.uni != 0, p.parts > 1, trace);
    return k ? march_launch_one(k, blocks, threads, march_mg_smem(p, threads), st, p) : (int)cudaErrorInvalidValue;
}

int march_mg_occupancy(int mode, bool uni, int threads, size_t smem) {
    const auto k = march_mg_fn(mode, uni, false, false);
    const int nb = k ? march_occupancy_one(k, threads, smem) : 0;
    return nb > 0 ? nb : 1;
}

int launch_march(int mode, const MarchParams &p, int blocks, int threads, void *stream, bool trace) {
    return launch_march_ex(mode, p, blocks, threads, stream, trace, false, false, false);
}

// ---------------------------------------------------------------------------
// Control variate preparation.  Y is the ray's contribution in the medium
// whose temperature and x_H2O are the mean of each wall-normal plane, with
// its flight through that medium replaced by a tabulated function of the
// ray's layer, spectral sample and wall-normal cosine mu:
//   J(mu) = the intensity the walk from the layer centre collects (same toll
//           cut-off, same wall emission as the 3-D march),
//   A(mu) = 1 - the transmissivity of its path out of the own layer,
// stored at the nodes u_m = m / kSurBins of u = sqrt(|mu|) per hemisphere and
// read by linear interpolation in u.  Whatever the table holds, its mean over
// the isotropic directions is a finite sum over the bins, so E[Y] per cell is
//   E[Y_a] = sum_s C_s k_i(s) (Ib_i(s) - Jhat_s(layer)),
//   E[Y_b] = sum_s C_s k_i(s) (Ib_i(s) - Ibar_s(layer)) Ahat_s(layer),
// exactly; the march tallies X - beta.Y and finalize adds beta.E[Y] back, so
// the estimate is unbiased for any beta and any table.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float cv_k(const CvParams &c, int sid, float T, float x) {
    int ti, xi = 0;
    float ft, fx = 0.f;
    grid_pos(T, c.T0, c.invdT, c.nT, &ti, &ft);
    if (c.mode == MODE_TX) {
        grid_pos(x, c.X0, c.invdX, c.nX, &xi, &fx);
        const float *s = c.ktab + (long long)sid * c.nT * c.nX + ti * c.nX + xi;
        const float k00 = __ldg(s), k01 = __ldg(s + 1);
        const float k10 = __ldg(s + c.nX), k11 = __ldg(s + c.nX + 1);
        const float k0 = fmaf(fx, k01 - k00, k00);
        const float k1 = fmaf(fx, k11 - k10, k10);
        return fmaf(ft, k1 - k0, k0);
    }
    const float *s = c.ktab + (long long)sid * c.nT + ti;
    const float k0 = __ldg(s), k1 = __ldg(s + 1);
    return fmaf(ft, k1 - k0, k0);
}

__device__ __forceinline__ float cv_ib(const CvParams &c, int band, float T) {
    int ti;
    float ft;
    grid_pos(T, c.T0, c.invdT, c.nT, &ti, &ft);
    const float *s = c.ibtab + band * c.nT + ti;
    const float i0 = __ldg(s), i1 = __ldg(s + 1);
    return fmaf(ft, i1 - i0, i0);
}

// (T_bar, x_bar) of every wall-normal plane, fixed-order reduction.
__global__ void cv_layer_kernel(const CvParams c) {
    const int w = blockIdx.x, f = blockIdx.y;
    const long long plane = (long long)c.na * c.nb;
    const long long base = ((long long)f * c.nw + w) * plane;
    __shared__ double sT[256], sX[256], sV[256];
    double aT = 0.0, aX = 0.0, aV = 0.0;
    for (long long i = threadIdx.x; i < plane; i += blockDim.x) {
        if (c.mode == MODE_TX) { const float2 v = c.fieldTX[base + i]; aT += v.x; aX += v.y; }
        else aT += c.fieldT[base + i];
        if (c.fieldV) aV += c.fieldV[base + i];
    }
    sT[threadIdx.x] = aT;
    sX[threadIdx.x] = aX;
    sV[threadIdx.x] = aV;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            sT[threadIdx.x] += sT[threadIdx.x + o];
            sX[threadIdx.x] += sX[threadIdx.x + o];
            sV[threadIdx.x] += sV[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        c.layer[(long long)f * c.nw + w] = make_float2((float)(sT[0] / plane), (float)(sX[0] / plane));
        if (c.layerV) c.layerV[(long long)f * c.nw + w] = (float)(sV[0] / plane);
    }
}

// Layer-mean absorption coefficient and band intensity per (field, sample, layer).
__global__ void cv_sur_kernel(const CvParams c) {
    const long long n = (long long)c.nfields * c.n_samples * c.nw;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        const int w = (int)(idx % c.nw);
        const long long fs = idx / c.nw;
        const int sid = (int)(fs % c.n_samples);
        const int f = (int)(fs / c.n_samples);
        const float2 L = c.layer[(long long)f * c.nw + w];
        float kb, Ib;
        if (c.mode == MODE_GREY) {
            const float t2 = L.x * L.x;
            kb = c.kappa;
            Ib = t2 * t2;
        } else {
            kb = cv_k(c, sid, L.x, L.y);
            Ib = cv_ib(c, sid / c.nq, L.x);
        }
        if (c.part) kb = fmaf(c.layerV[(long long)f * c.nw + w], c.part[c.mode == MODE_GREY ? 0 : sid / c.nq].x, kb);
        c.sur[idx] = make_float2(kb, Ib);
    }
}

// Surrogate table and its exact means, one block per (field, sample).  The
// surrogate ray leaves the centre o_l of layer l with wall-normal cosine mu
// and flies straight through the layers of constant (k, Ib) = sur[l] to the
// black wall (intensity Iw); what it collects is
//   J_l = (1 - e^{-h_l}) Ib_l + e^{-h_l} F_{l+1}   (east; west alike),
// with h_l = k_l (f_{l+1} - o_l) / mu its own half-layer depth and F_i the
// intensity collected by a ray entering layer i from the west face,
//   F_i = (1 - e^{-d_i}) Ib_i + e^{-d_i} F_{i+1},  F_nw = Iw,  d_i = k_i (f_{i+1} - f_i) / mu,
// and its own-layer absorptance is A_l = 1 - e^{-h_l}.  So one sweep per
// (node, hemisphere) from the far wall gives every layer's node: thread
// (h, m) sweeps mu = u_m^2 (u_m = m / kSurBins; the node u = 0 at mu =
// 2^-30, the grazing limit) across the layers, one layer per step, with
// e^{-x} - 1 = mc_expm1(-x):
//   J = F + e1h (F - Ib_l),  A = -e1h,  then  F <- F + e1 (F - Ib_l).
// After each step the block writes the two layers' bins (J0, dJ, A0, dA)
// and their contributions to the means: with mu uniform on [0, 1] per
// hemisphere, u has density 2u, and bin m contributes
//   E_h[J] += ((2m + 1) J0 + (m + 2/3) dJ) / kSurBins^2
//          = (3 (2m + 1) J0 + (3m + 2) dJ) / (3 kSurBins^2),
// likewise for A.  The integer-weighted terms are formed exactly as
// float pairs (the product's rounding error by fma) and summed as float
// pairs (error-free sums), each hemisphere's 64 terms by two warps in
// butterfly order, then in FP64: about 48 bits, at FP32 rates (this GPU's
// FP64 rate is a small fraction of that).
constexpr int kSurNodes = kSurBins + 1;

// (hi, lo) float pairs: ff_add (mc_march.cuh) sums two of them
// w * v as an exact pair (w a small integer)
__device__ __forceinline__ float2 ff_mul(float w, float v) {
    const float p = w * v;
    return make_float2(p, fmaf(w, v, -p));
}
constexpr int kTableThreads = 160;  // 2 kSurNodes sweeps; 2 kSurBins bins
size_t cv_table_smem(int nw) { return (size_t)nw * (2 * sizeof(double2) + sizeof(float2) + sizeof(float)) + 16; }

__global__ void __launch_bounds__(kTableThreads) cv_table_kernel(const CvParams c) {
    extern __shared__ double2 s_mean[];                    // [nw][2] per-hemisphere sums (eJ, eA)
    float2 *s_sur = reinterpret_cast<float2 *>(s_mean + 2 * c.nw);  // [nw] (k, Ib)
    float *s_fw = reinterpret_cast<float *>(s_sur + c.nw);  // [nw + 1] faces
    __shared__ float2 s_val[2][kSurNodes];                 // this step's nodes (J, A)
    __shared__ double2 s_half[4];                          // this step's warp sums
    const int t = threadIdx.x, nw = c.nw;
    const long long fs = blockIdx.x;                       // field * n_samples + sample
    const int sid = (int)(fs % c.n_samples);
    const int band = c.mode == MODE_GREY ? 0 : sid / c.nq;
    const float2 *sp = c.sur + fs * nw;
    for (int i = t; i < nw; i += kTableThreads) s_sur[i] = sp[i];
    for (int i = t; i <= nw; i += kTableThreads) s_fw[i] = c.fw[i];
    // sweep thread: hemisphere h (0: towards the west wall), node m
    const int h = t >= kSurNodes ? 1 : 0, m = t - h * kSurNodes;
    float invmu = 0.0f, F = 0.0f;
    if (t < 2 * kSurNodes) {
        const float u = (float)m * (1.0f / (float)kSurBins);
        const float mu = m ? u * u : 9.31322574615478516e-10f;  // 2^-30
        invmu = 1.0f / mu;
        F = c.mode == MODE_GREY ? c.Tw4[h] : __ldg(c.ibw + h * c.nbands + band);
    }
    __syncthreads();
    for (int step = 0; step < nw; ++step) {
        if (t < 2 * kSurNodes) {
            const int l = h ? nw - 1 - step : step;
            const float2 kv = s_sur[l];
            const float f0 = s_fw[l], f1 = s_fw[l + 1];
            const float o = (f0 + f1) * 0.5f;
            const float half = h ? (f1 - o) * invmu : (o - f0) * invmu;
            const float e1h = mc_expm1(-(kv.x * half));
            s_val[h][m] = make_float2(fmaf(e1h, F - kv.y, F), -e1h);
            const float e1 = mc_expm1(-(kv.x * ((f1 - f0) * invmu)));
            F = fmaf(e1, F - kv.y, F);
        }
        __syncthreads();
        if (t < 2 * kSurBins) {
            const int hb = t / kSurBins, mb = t - hb * kSurBins;
            const int l = hb ? nw - 1 - step : step;
            const float2 v0 = s_val[hb][mb], v1 = s_val[hb][mb + 1];
            const float dJ = v1.x - v0.x, dA = v1.y - v0.y;
            c.surtab[(fs * nw + l) * (2 * kSurBins) + t] = make_float4(v0.x, dJ, v0.y, dA);
            const float w0 = (float)(3 * (2 * mb + 1)), w1 = (float)(3 * mb + 2);
            float2 eJ = ff_add(ff_mul(w0, v0.x), ff_mul(w1, dJ));
            float2 eA = ff_add(ff_mul(w0, v0.y), ff_mul(w1, dA));
            for (int o = 16; o > 0; o >>= 1) {
                float2 pJ, pA;
                pJ.x = __shfl_xor_sync(0xffffffffu, eJ.x, o);
                pJ.y = __shfl_xor_sync(0xffffffffu, eJ.y, o);
                pA.x = __shfl_xor_sync(0xffffffffu, eA.x, o);
                pA.y = __shfl_xor_sync(0xffffffffu, eA.y, o);
                eJ = ff_add(eJ, pJ);
                eA = ff_add(eA, pA);
            }
            if ((t & 31) == 0)
                s_half[t >> 5] = make_double2((double)eJ.x + (double)eJ.y, (double)eA.x + (double)eA.y);
        }
        __syncthreads();
        if (t < 2) {  // the step's two layers
            const int l = t ? nw - 1 - step : step;
            s_mean[2 * l + t] = make_double2(s_half[2 * t].x + s_half[2 * t + 1].x,
                                             s_half[2 * t].y + s_half[2 * t + 1].y);
        }
    }
    __syncthreads();
    // both hemispheres, weight 1/2; the sums carry the factor 3
    const double sc = 0.5 / (3.0 * (double)kSurBins * (double)kSurBins);
    for (int l = t; l < nw; l += kTableThreads) {
        const double2 a = s_mean[2 * l], b = s_mean[2 * l + 1];
        const double J = (a.x + b.x) * sc, A = (a.y + b.y) * sc;
        const long long idx = fs * nw + l;
        c.Jhat[idx] = make_double2(J, A);
    }
}

// E[Y] of the grey model per (field, cell of the region), tally layout:
//   E[Y_a] = W (T^4 - Jhat(layer)),  E[Y_b] = W (T^4 - Ibar(layer)) Ahat(layer),
// W the march's weight 4 sigma (kappa + fv a).
__global__ void cv_mean_grey_kernel(const CvParams c) {
    const int njR = c.ea1 - c.ea0, nkR = c.eb1 - c.eb0;
    const long long n = (long long)c.nfields * c.region_cells;
    const long long plane = (long long)c.na * c.nb;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        const int f = (int)(idx / c.region_cells);
        const long long tc = idx - (long long)f * c.region_cells;
        const int jR = (int)(tc % njR);
        const long long r = tc / njR;
        const int kR = (int)(r % nkR);
        const int w = c.ew0 + (int)(r / nkR);
        const long long cell = ((long long)f * c.nw + w) * plane + (long long)(c.eb0 + kR) * c.na + (c.ea0 + jR);
        const float T = c.fieldT[cell], t2 = T * T;
        const long long sbase = (long long)f * c.n_samples * c.nw + w;
        const double2 jh = c.Jhat[sbase];
        // the march's own FP32 weight when particles are present
        const double Wk = c.part ? (double)((float)(4.0 * 5.670373e-08) * fmaf(c.fieldV[cell], c.part[0].x, c.kappa)) : c.Wgrey;
        c.muY[(long long)f * c.n_groups * c.region_cells + tc] =
            make_double2(Wk * ((double)(t2 * t2) - jh.x), Wk * ((double)(t2 * t2) - (double)c.sur[sbase].y) * jh.y);
    }
}

// ---------------------------------------------------------------------------
// E[Y] through node sums (tables).  With k_s(T, x) the
// bilinear and Ib_s(T) the linear interpolant of the tables at the cell's
// table coordinates (weights wt_a in T, wx_b in x; sum_a' wt_a' = 1),
//   E[Y_a] = sum_s C_s k_s (Ib_s - Jhat_s(w))
//          = sum_{b,a,a'} wx_b wt_a wt_a' Da(w)[t][x_b][a][a'],
//   E[Y_b] = sum_s C_s Ahat_s(w) k_s (Ib_s - Ibar_s(w))
//          = sum_{b,a,a'} wx_b wt_a wt_a' Db(w)[t][x_b][a][a'],
// with the node sums per (field, group, layer) and table cell (t, x)
//   Da[t][x][a][a'] = sum_s C_s k_s[t+a][x] (Ib_s[t+a'] - Jhat_s),
//   Db[t][x][a][a'] = sum_s C_s Ahat_s k_s[t+a][x] (Ib_s[t+a'] - Ibar_s):
// a cell needs 16 node sums per group instead of a pass over the group's
// samples, and the differences Ib - Jhat, where optically thick samples
// cancel, are formed per sample before any sum.  Particles add fv a_s to k_s:
// four more sums per table temperature, with a_s for the k of the node,
//   Pa[t][a'] = sum_s C_s a_s (Ib_s[t+a'] - Jhat_s),  Pb alike,
// of which a cell takes fv sum_a' wt_a' P[t][a'] (96^3 cells, 8 groups of 128
// samples: 4.19 ms a pass over the samples, 0.63 ms both kernels of the sums).  Arithmetic in float pairs
// (hi + lo, about 48 bits: error-free products by fma and error-free sums;
// this file is compiled without FMA contraction), at FP32 rates -- this
// GPU's FP64 rate is a small fraction of them.  The cell's weights are
// formed in FP64 and its 16-term combination summed in pairs.
// ---------------------------------------------------------------------------
struct NodeLayout {
    // table cells (t, x), work units (one per cell, with particles one more
    // per temperature), pairs per (field, group, layer): Da then Db, 4 each
    // per cell, then (Pa, Pb), 2 each per temperature
    int nTc, units, per;
};
__host__ __device__ inline NodeLayout node_layout(const CvParams &c) {
    NodeLayout L;
    L.nTc = (c.nT - 1) * c.nX;
    L.units = L.nTc + (c.part ? c.nT - 1 : 0);
    L.per = L.nTc * 8 + (L.units - L.nTc) * 4;
    return L;
}

long long cv_node_count(const CvParams &c) {
    const NodeLayout L = node_layout(c);
    const long long niR = c.ew1 - c.ew0;
    return (long long)c.nfields * c.n_groups * niR * L.per;
}

// a double as a float pair
__device__ __forceinline__ float2 ff_of(double v) {
    const float hi = (float)v;
    return make_float2(hi, (float)(v - (double)hi));
}
// a pair times a float (the low part's product rounded)
__device__ __forceinline__ float2 ff_mulf(float2 a, float b) {
    const float p = a.x * b;
    return make_float2(p, fmaf(a.x, b, -p) + a.y * b);
}
// a pair times a pair
__device__ __forceinline__ float2 ff_mulff(float2 a, float2 b) {
    const float p = a.x * b.x;
    return make_float2(p, fmaf(a.x, b.x, -p) + (a.x * b.y + a.y * b.x));
}
// a float minus a pair, as a pair
__device__ __forceinline__ float2 ff_fsub(float a, float2 b) { return ff_add(make_float2(a, 0.0f), make_float2(-b.x, -b.y)); }

// Blocks: (field, group, region layer).  Work units: the table cells (t, x),
// each with its eight sums, one per thread in rounds of blockDim.  The
// per-sample weights and the inputs of the differences come from shared
// memory in chunks of 256 samples.
__global__ void __launch_bounds__(256) cv_nodes_kernel(const CvParams c) {
    __shared__ int s_ib[256];      // band * nT
    __shared__ int s_koff[256];    // sample * nT * nX
    __shared__ float2 s_C[256], s_CA[256], s_J[256];  // C, C Ahat, Jhat as pairs
    __shared__ float s_Ibar[256], s_part[256];
    const NodeLayout L = node_layout(c);
    const int niR = c.ew1 - c.ew0;
    const long long b = blockIdx.x;
    const int wR = (int)(b % niR);
    const long long fg = b / niR;
    const int g = (int)(fg % c.n_groups);
    const int f = (int)(fg / c.n_groups);
    const int w = c.ew0 + wR;
    float2 *out = reinterpret_cast<float2 *>(c.nodes) + b * L.per;
    const int q0 = c.grp_start[g], q1 = c.grp_start[g + 1];
    for (int u0 = 0; u0 < L.units; u0 += blockDim.x) {
        const int u = u0 + threadIdx.x;
        const bool particles = u >= L.nTc;
        const int t = particles ? u - L.nTc : u / c.nX, x = particles ? 0 : u - t * c.nX;
        float2 acc[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = make_float2(0.0f, 0.0f);
        for (int qc = q0; qc < q1; qc += 256) {
            const int nq = min(256, q1 - qc);
            __syncthreads();
            if ((int)threadIdx.x < nq) {
                const int q = qc + threadIdx.x;
                const int sid = c.samp_id[q];
                const double C = c.samp_C[q];
                const long long o = ((long long)f * c.n_samples + sid) * c.nw + w;
                const double2 jh = c.Jhat[o];
                s_ib[threadIdx.x] = (sid / c.nq) * c.nT;
                s_koff[threadIdx.x] = sid * c.nT * c.nX;
                s_C[threadIdx.x] = ff_of(C);
                s_CA[threadIdx.x] = ff_of(C * jh.y);
                s_J[threadIdx.x] = ff_of(jh.x);
                s_Ibar[threadIdx.x] = c.sur[o].y;
                s_part[threadIdx.x] = c.part ? c.part[sid / c.nq].x : 0.0f;
            }
            __syncthreads();
            if (u >= L.units) continue;
            for (int j = 0; j < nq; ++j) {
                const float *kk = c.ktab + s_koff[j] + t * c.nX + x;
                const float *ib = c.ibtab + s_ib[j] + t;
                const float k0 = particles ? s_part[j] : __ldg(kk), k1 = __ldg(kk + c.nX);
                const float i0 = __ldg(ib), i1 = __ldg(ib + 1);
                const float2 J = s_J[j];
                const float Ibar = s_Ibar[j];
                const float2 da0 = ff_fsub(i0, J), da1 = ff_fsub(i1, J);
                const float2 db0 = ff_fsub(i0, make_float2(Ibar, 0.0f)), db1 = ff_fsub(i1, make_float2(Ibar, 0.0f));
                const float2 ck0 = ff_mulf(s_C[j], k0), ck1 = ff_mulf(s_C[j], k1);
                const float2 ca0 = ff_mulf(s_CA[j], k0), ca1 = ff_mulf(s_CA[j], k1);
                acc[0] = ff_add(acc[0], ff_mulff(ck0, da0));
                acc[1] = ff_add(acc[1], ff_mulff(ck0, da1));
                acc[2] = ff_add(acc[2], ff_mulff(ck1, da0));
                acc[3] = ff_add(acc[3], ff_mulff(ck1, da1));
                acc[4] = ff_add(acc[4], ff_mulff(ca0, db0));
                acc[5] = ff_add(acc[5], ff_mulff(ca0, db1));
                acc[6] = ff_add(acc[6], ff_mulff(ca1, db0));
                acc[7] = ff_add(acc[7], ff_mulff(ca1, db1));
            }
        }
        if (u < L.nTc) {  // layout: Da [t][x][a*2 + a'], then Db alike
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                out[(long long)u * 4 + r] = acc[r];
                out[(long long)L.nTc * 4 + (long long)u * 4 + r] = acc[4 + r];
            }
        } else if (particles && u < L.units) {
            float2 *o = out + (long long)L.nTc * 8 + (long long)t * 4;
            o[0] = acc[0]; o[1] = acc[1]; o[2] = acc[4]; o[3] = acc[5];
        }
    }
}

// E[Y] per (field, cell) from the node sums, all groups.
__global__ void cv_mean_nodes_kernel(const CvParams c) {
    const NodeLayout L = node_layout(c);
    const int njR = c.ea1 - c.ea0, nkR = c.eb1 - c.eb0, niR = c.ew1 - c.ew0;
    const long long n = (long long)c.nfields * c.region_cells;
    const long long plane = (long long)c.na * c.nb;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
         idx += (long long)gridDim.x * blockDim.x) {
        const int f = (int)(idx / c.region_cells);
        const long long tc = idx - (long long)f * c.region_cells;
        const int jR = (int)(tc % njR);
        const long long r = tc / njR;
        const int kR = (int)(r % nkR);
        const int iR = (int)(r / nkR);
        const long long cell = (long long)f * c.nw * plane + (long long)(c.ew0 + iR) * plane +
                               (long long)(c.eb0 + kR) * c.na + (c.ea0 + jR);
        float T, x = 0.f;
        if (c.mode == MODE_TX) { const float2 v = c.fieldTX[cell]; T = v.x; x = v.y; }
        else T = c.fieldT[cell];
        int ti, xi = 0;
        float ftf, fxf = 0.f;
        grid_pos(T, c.T0, c.invdT, c.nT, &ti, &ftf);
        if (c.mode == MODE_TX) grid_pos(x, c.X0, c.invdX, c.nX, &xi, &fxf);
        const double ft = ftf, fx = fxf;
        const double wt[2] = {1.0 - ft, ft};
        const double wx[2] = {1.0 - fx, fx};
        const int nb = c.nX > 1 ? 2 : 1;
        // the cell's interpolation weights w4[bx][a][a'] = wx[bx] wt[a] wt[a']
        // (the product of the k and Ib interpolations), formed once for all
        // groups
        float2 w4[2][4];
        for (int bx = 0; bx < nb; ++bx)
            for (int a = 0; a < 2; ++a)
                for (int a2 = 0; a2 < 2; ++a2) w4[bx][a * 2 + a2] = ff_of(wx[bx] * wt[a] * wt[a2]);
        float2 wp[2];
        if (c.part) {
            const double fv = c.fieldV[cell];
            wp[0] = ff_of(fv * wt[0]);
            wp[1] = ff_of(fv * wt[1]);
        }
        for (int g = 0; g < c.n_groups; ++g) {
            const float2 *lay = reinterpret_cast<const float2 *>(c.nodes) +
                                (((long long)f * c.n_groups + g) * niR + iR) * L.per;
            float2 ea = make_float2(0.0f, 0.0f), eb = make_float2(0.0f, 0.0f);
            for (int bx = 0; bx < nb; ++bx) {
                const long long o = ((long long)ti * c.nX + xi + bx) * 4;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    ea = ff_add(ea, ff_mulff(w4[bx][q], __ldg(lay + o + q)));
                    eb = ff_add(eb, ff_mulff(w4[bx][q], __ldg(lay + (long long)L.nTc * 4 + o + q)));
                }
            }
            if (c.part) {
                const float2 *o = lay + (long long)L.nTc * 8 + (long long)ti * 4;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    ea = ff_add(ea, ff_mulff(wp[q], __ldg(o + q)));
                    eb = ff_add(eb, ff_mulff(wp[q], __ldg(o + 2 + q)));
                }
            }
            c.muY[((long long)f * c.n_groups + g) * c.region_cells + tc] =
                make_double2((double)ea.x + (double)ea.y, (double)eb.x + (double)eb.y);
        }
    }
}

// One warp per packet: lane l takes the packet's cells l, l + 32, ...
__global__ void adaptive_rays_kernel(const AdaptParams A) {
    const int lane = threadIdx.x & 31;
    const long long wid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long plane = (long long)A.na * A.nb;
    for (long long p = wid; p < A.n_packets; p += nwarp) {
        const int pa = (int)(p % A.npa);
        const long long rest = p / A.npa;
        const int pb = (int)(rest % A.npb), pw = (int)(rest / A.npb);
        float tsum = 0.0f, cnt = 0.0f;
        for (int cl = lane; cl < A.tile_a * A.tile_b; cl += 32) {
            const int jR = pa * A.tile_a + cl % A.tile_a, kR = pb * A.tile_b + cl / A.tile_a;
            if (jR >= A.njR || kR >= A.nkR) continue;
            const int i = A.ew0 + pw;
            const float h = cbrtf((A.fw[i + 1] - A.fw[i]) * A.da * A.db);
            for (int f = 0; f < A.nfields; ++f) {
                const long long cell = f * A.field_stride + i * plane + (long long)(A.eb0 + kR) * A.na + (A.ea0 + jR);
                float kp = A.kappa;
                if (A.kP) {
                    int ti, xi = 0;
                    float ft, fx = 0.0f;
                    if (A.mode == MODE_TX) {
                        const float2 v = A.fTX[cell];
                        grid_pos(v.x, A.T0, A.invdT, A.nT, &ti, &ft);
                        grid_pos(v.y, A.X0, A.invdX, A.nX, &xi, &fx);
                    } else {
                        grid_pos(A.fT[cell], A.T0, A.invdT, A.nT, &ti, &ft);
                    }
                    const float *k = A.kP + ti * A.nX + xi;
                    const float dx = (A.nX > 1) ? 1.0f : 0.0f;
                    const float k00 = k[0], k01 = A.nX > 1 ? k[1] : k[0];
                    const float k10 = k[A.nX], k11 = A.nX > 1 ? k[A.nX + 1] : k[A.nX];
                    const float a0 = k00 + fx * dx * (k01 - k00), a1 = k10 + fx * dx * (k11 - k10);
                    kp = a0 + ft * (a1 - a0);
                }
                tsum += kp * h;
                cnt += 1.0f;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            tsum += __shfl_xor_sync(0xffffffffu, tsum, o);
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
        if (lane == 0) {
            const float x = A.per_tau * (cnt > 0.0f ? tsum / cnt : 0.0f);
            int r = (int)rintf(x / (float)A.B) * A.B;
            r = min(max(r, A.nmin), A.nmax);
            A.rays[p] = r;
        }
    }
}

int launch_adaptive_rays(const AdaptParams &a, void *stream) {
    const long long threads = (long long)a.n_packets * 32;
    dnsmc::note_launch();
    adaptive_rays_kernel<<<grid_for(threads, 256), 256, 0, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

// Longest-first queue order.  Bucket of an item = min(rays / B, buckets - 1),
// counted in descending bucket order; items of one bucket keep no particular
// order (results do not depend on the processing order).
__global__ void order_hist_kernel(const int *rays, int gstride, int n_packets, int n_groups, long long n_items, int B,
                                  unsigned int *hist) {
    const long long per_field = (long long)n_groups * n_packets;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_items;
         i += (long long)gridDim.x * blockDim.x) {
        const long long gp = i % per_field;
        const int g = (int)(gp / n_packets), p = (int)(gp % n_packets);
        const int b = min(rays[g * gstride + p] / B, kOrderBuckets - 1);
        atomicAdd(hist + (kOrderBuckets - 1 - b), 1u);
    }
}

// exclusive scan of the kOrderBuckets counts in place (one block of 1024)
__global__ void order_scan_kernel(unsigned int *hist) {
    __shared__ unsigned int part[1024];
    constexpr int per = kOrderBuckets / 1024;
    const int t = threadIdx.x;
    unsigned int loc[per], run = 0;
    for (int q = 0; q < per; ++q) { loc[q] = hist[t * per + q]; run += loc[q]; }
    part[t] = run;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned int v = t >= o ? part[t - o] : 0u;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    unsigned int base = t ? part[t - 1] : 0u;
    for (int q = 0; q < per; ++q) { const unsigned int v = loc[q]; hist[t * per + q] = base; base += v; }
}

__global__ void order_scatter_kernel(const int *rays, int gstride, int n_packets, int n_groups, long long n_items,
                                     int B, unsigned int *hist, unsigned int *order) {
    const long long per_field = (long long)n_groups * n_packets;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n_items;
         i += (long long)gridDim.x * blockDim.x) {
        const long long gp = i % per_field;
        const int g = (int)(gp / n_packets), p = (int)(gp % n_packets);
        const int b = min(rays[g * gstride + p] / B, kOrderBuckets - 1);
        const unsigned int pos = atomicAdd(hist + (kOrderBuckets - 1 - b), 1u);
        order[pos] = (unsigned int)i;
    }
}

int launch_item_order(const int *rays, int gstride, int n_packets, int n_groups, long long n_items, int B,
                      unsigned int *hist, unsigned int *order, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(hist, 0, kOrderBuckets * sizeof(unsigned int), st);
    if (e != cudaSuccess) return (int)e;
    dnsmc::note_launch();
    order_hist_kernel<<<grid_for(n_items, 256), 256, 0, st>>>(rays, gstride, n_packets, n_groups, n_items, B, hist);
    dnsmc::note_launch();
    order_scan_kernel<<<1, 1024, 0, st>>>(hist);
    dnsmc::note_launch();
    order_scatter_kernel<<<grid_for(n_items, 256), 256, 0, st>>>(rays, gstride, n_packets, n_groups, n_items, B,
                                                                 hist, order);
    return (int)cudaGetLastError();
}

int launch_cv_prepare(const CvParams &c, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    dnsmc::note_launch();
    cv_layer_kernel<<<dim3(c.nw, c.nfields), 256, 0, st>>>(c);
    const long long n = (long long)c.nfields * c.n_samples * c.nw;
    dnsmc::note_launch();
    cv_sur_kernel<<<grid_for(n, 256), 256, 0, st>>>(c);
    dnsmc::note_launch();
    // one block per (field, sample); its shared memory beyond 48 KB was
    // allowed once per device (cv_table_allow_smem), outside any capture
    const size_t smem = cv_table_smem(c.nw);
    cv_table_kernel<<<(unsigned)((long long)c.nfields * c.n_samples), kTableThreads, smem, st>>>(c);
    return (int)cudaGetLastError();
}

// The table kernel's dynamic shared memory for the largest grid the control
// variate takes (imax 4096), set once per device.
int cv_table_allow_smem() {
    return (int)cudaFuncSetAttribute(cv_table_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)cv_table_smem(kCvMaxPlanes));
}

int launch_cv_mean(const CvParams &c, void *stream) {
    const long long n = (long long)c.nfields * c.region_cells;
    cudaStream_t st = (cudaStream_t)stream;
    if (c.nodes) {  // tables: node sums, then the cells
        const long long blocks = (long long)c.nfields * c.n_groups * (c.ew1 - c.ew0);
        dnsmc::note_launch();
        cv_nodes_kernel<<<(unsigned)blocks, 256, 0, st>>>(c);
        dnsmc::note_launch();
        cv_mean_nodes_kernel<<<grid_for(n, 256), 256, 0, st>>>(c);
    } else {
        dnsmc::note_launch();
        cv_mean_grey_kernel<<<grid_for(n, 256), 256, 0, st>>>(c);
    }
    return (int)cudaGetLastError();
}

int launch_field_pos(const FieldPos &q, void *stream) {
    const long long n = (long long)q.nfields * q.nw * q.pnb * q.pna;
    dnsmc::note_launch();
    field_pos_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(q);
    return (int)cudaGetLastError();
}

// (1/N, 1/(N-1)) of every ray count (0 where undefined)
__global__ void ray_reciprocals_kernel(const int *rays, long long n, double2 *out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int N = rays[i];
        out[i] = make_double2(N > 0 ? 1.0 / N : 0.0, N > 1 ? 1.0 / (N - 1) : 0.0);
    }
}

static double2 reciprocals(int N) { return make_double2(N > 0 ? 1.0 / N : 0.0, N > 1 ? 1.0 / (N - 1) : 0.0); }

int launch_finalize(const FinalizeParams &p, void *stream) {
    FinalizeParams q = p;
    q.rcp_uniform = reciprocals(p.rays);
    q.rcp_batch = reciprocals(p.nbatch);
    cudaStream_t st = (cudaStream_t)stream;
    if (q.rays_per_packet) {
        if (!q.rcp) return (int)cudaErrorInvalidValue;
        const long long nr = finalize_rcp_count(q);
        dnsmc::note_launch();
        ray_reciprocals_kernel<<<grid_for(nr, 256), 256, 0, st>>>(q.rays_per_packet, nr, q.rcp);
    }
    const unsigned tiles = (unsigned)(((q.njR + kFinTile - 1) / kFinTile) * ((q.niR + kFinTile - 1) / kFinTile));
    if (tiles == 0 || q.nkR <= 0 || q.nfields <= 0) return (int)cudaGetLastError();
    dnsmc::note_launch();
    finalize_kernel<<<dim3(tiles, (unsigned)q.nkR, (unsigned)q.nfields), kFinTile * kFinRows, 0, st>>>(q);
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Spline coarsening of the temperature for the multigrid march: the
// reference's interp3D (code/spline.cpp:35-116), a separable natural cubic
// spline through the fine cell centres along x, then y, then z, evaluated at
// the coarse cell centres.  The arithmetic is the Numerical Recipes spline /
// splint of code/spline.cpp:119-170 written as the oracle restates it (float
// with the same double sub-expressions; this translation unit is compiled
// with -fmad=false), so the coarse fields are bit-identical to the oracle's.
//
// What bounds it is the tridiagonal recurrence of a line, n dependent steps
// in FP64.  Everything that is not in that chain is taken out of it: the
// coefficients that depend on positions alone come from the host, the right
// sides and the evaluation are spread over the block, and the chain's
// division by p is q0 = a * r, q = fma(fma(-q0, p, a), r, q0) with r = RN(1/p)
// (Markstein 1990).  q is the correctly rounded a / p here: a - q0 p is exact
// (p has 24 bits), so before its rounding q differs from a / p by 2^-52 of an
// ulp at most, while a quotient by a 24-bit p keeps 2^-25 of an ulp from every
// midpoint of doubles.  All levels and fields share a launch, and the pass
// along x one recurrence for all levels: three launches.  64^3, four coarse
// levels: 99 us (twelve launches, a thread per line with its chain in
// global memory: 1250 us).
// ---------------------------------------------------------------------------
template <bool WORK>
__global__ void __launch_bounds__(256) spline_pass_kernel(const SplinePass q) {
    extern __shared__ double s_line[];
    const int W = q.lines, W1 = W + 1, n = q.n;
    int j = 0;
    while (j + 1 < q.njobs && (int)blockIdx.x >= q.job[j + 1].block0) ++j;
    const SplineJob &b = q.job[j];
    const long long L0 = (long long)((int)blockIdx.x - b.block0) * W;
    const int nl = (int)min((long long)W, b.nlines - L0);  // this block's lines
    // [element][line]: right side, then u, then the second derivative; value
    double *t = WORK ? q.work + (size_t)(blockIdx.y * (size_t)gridDim.x + blockIdx.x) * spline_line_doubles(n, W) : s_line;
    float *a = reinterpret_cast<float *>(t + (size_t)n * W1);
    auto slot = [&](int e, int l) { return reinterpret_cast<float *>(t + (size_t)e * W1 + l); };
    for (int f = blockIdx.y; f < q.nfields; f += gridDim.y) {
        const float *src = b.src + f * b.s_f;
        for (int k = threadIdx.x; k < n * nl; k += blockDim.x) {
            int e, l;
            if (b.s_e == 1) { l = k / n; e = k - l * n; } else { e = k / nl; l = k - e * nl; }
            const unsigned lb = (unsigned)(L0 + l) / b.na, la = (unsigned)(L0 + l) - lb * b.na;
            a[(size_t)e * W1 + l] = src[(la * b.s_a + lb * b.s_b + e * b.s_e) * q.src_step];
        }
        __syncthreads();
        for (int k = threadIdx.x; k < (n - 2) * nl; k += blockDim.x) {
            const int e = k / nl + 1, l = k - (e - 1) * nl;
            const float *v = a + (size_t)e * W1 + l;
            const float ui = (v[W1] - v[0]) / (q.x[e + 1] - q.x[e]) - (v[0] - v[-W1]) / (q.x[e] - q.x[e - 1]);
            t[(size_t)e * W1 + l] = 6.0 * ui / (q.x[e + 1] - q.x[e - 1]);
        }
        __syncthreads();
        if ((int)threadIdx.x < nl) {
            const int l = threadIdx.x;
            float u = 0.0f;
            *slot(0, l) = 0.0f;
#pragma unroll 4
            for (int e = 1; e < n - 1; ++e) {
                const SplineCoef k = q.coef[e];
                const double num = t[(size_t)e * W1 + l] - k.sig * u;
                const double q0 = num * k.rp;
                const double q1 = fma(fma(-q0, k.p, num), k.rp, q0);
                const bool fin = (__double2hiint(num) & 0x7ff00000) != 0x7ff00000;
                u = (float)(fin ? q1 : num);  // p > 0: an infinity stays one
                *slot(e, l) = u;
            }
            float y2 = 0.0f;
            *slot(n - 1, l) = 0.0f;
#pragma unroll 4
            for (int e = n - 2; e >= 0; --e) {
                y2 = q.coef[e].c * y2 + *slot(e, l);
                *slot(e, l) = y2;
            }
        }
        __syncthreads();
        for (int o = b.out0; o < b.out0 + b.nout; ++o) {
            const SplineOut &w = q.out[o];
            float *dst = w.dst + f * w.d_f;
            for (int k = threadIdx.x; k < w.m * nl; k += blockDim.x) {
                int c, l;
                if (w.d_e == 1) { l = k / w.m; c = k - l * w.m; } else { c = k / nl; l = k - c * nl; }
                const SplineAt p = w.at[c];
                const float *v = a + (size_t)p.lo * W1 + l;
                const float y2lo = *slot(p.lo, l), y2hi = *slot(p.lo + 1, l);
                const unsigned lb = (unsigned)(L0 + l) / b.na, la = (unsigned)(L0 + l) - lb * b.na;
                dst[la * w.d_a + lb * w.d_b + c * w.d_e] =
                    (float)(p.aa * v[0] + p.bb * v[W1] +
                            ((p.aa * p.aa * p.aa - p.aa) * y2lo + (p.bb * p.bb * p.bb - p.bb) * y2hi) * p.h2 / 6.0);
            }
        }
        __syncthreads();
    }
}

// Lines of a block: 32, fewer where that leaves SMs without a block (the
// chain's time does not depend on it) or the lines do not fit in shared
// memory; lines too long for it even so stay in q.work.
int launch_spline_pass(SplinePass &q, void *stream) {
    const size_t limit = 200u * 1024u;
    long long lines = 0;
    for (int j = 0; j < q.njobs; ++j) lines += q.job[j].nlines;
    q.lines = 32;
    while (q.lines > 8 && lines * q.nfields < 152ll * q.lines) q.lines /= 2;
    while (q.lines > 1 && spline_line_doubles(q.n, q.lines) * sizeof(double) > limit) q.lines /= 2;
    const size_t smem = spline_line_doubles(q.n, q.lines) * sizeof(double);
    const bool work = smem > limit;
    long long blocks = 0;
    for (int j = 0; j < q.njobs; ++j) {
        q.job[j].block0 = (int)blocks;
        blocks += (q.job[j].nlines + q.lines - 1) / q.lines;
    }
    if (blocks <= 0 || q.nfields <= 0) return 0;
    const dim3 grid((unsigned)blocks, (unsigned)(work ? 1 : std::min(q.nfields, 65535)));
    dnsmc::note_launch();
    if (work) {
        if (!q.work) return (int)cudaErrorInvalidValue;
        spline_pass_kernel<true><<<grid, 256, 0, (cudaStream_t)stream>>>(q);
    } else {
        if (smem > 48u * 1024u) {
            const cudaError_t e = cudaFuncSetAttribute(spline_pass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
            if (e != cudaSuccess) return (int)e;
        }
        spline_pass_kernel<false><<<grid, 256, smem, (cudaStream_t)stream>>>(q);
    }
    return (int)cudaGetLastError();
}

int launch_pack_T(const float *src, float *dst, int nw, int na, int nb, long long si, long long sj,
                  long long sk, long long base, void *stream) {
    const long long n = (long long)nw * na * nb;
    dnsmc::note_launch();
    pack_T_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, nw, na, nb, si, sj, sk, base);
    return (int)cudaGetLastError();
}

int launch_pack_T4(const float *src, float *dst, int nw, int na, int nb, int pna, int pnb, void *stream) {
    const long long n = (long long)nw * pna * pnb;
    dnsmc::note_launch();
    pack_T4_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, nw, na, nb, pna, pnb);
    return (int)cudaGetLastError();
}

int launch_pack_TX(const float *srcT, const float *srcX, float2 *dst, int nw, int na, int nb, long long si,
                   long long sj, long long sk, long long base, void *stream) {
    const long long n = (long long)nw * na * nb;
    dnsmc::note_launch();
    pack_TX_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(srcT, srcX, dst, nw, na, nb, si, sj, sk, base);
    return (int)cudaGetLastError();
}

int launch_slabs(const float *k, const float *ib, float2 *slab, int nS, int nq, int nT, int nX, int klen, int len, void *stream) {
    if (nS <= 0 || len <= 0) return 0;
    dnsmc::note_launch();
    slab_kernel<<<grid_for((long long)nS * len, 256), 256, 0, (cudaStream_t)stream>>>(k, ib, slab, nS, nq, nT, nX, klen, len);
    return (int)cudaGetLastError();
}
int launch_pack_stats(const float *srcT, const float *srcX, float *dst, int nw, int na, int nb, long long si, long long sj,
                      long long sk, long long base, double *partials, double *out, void *stream) {
    const unsigned n = (unsigned)((long long)nw * na * nb);
    const unsigned blocks = std::min((unsigned)kStatBlocks, (n + kStatThreads - 1) / kStatThreads);
    FieldStats *part = reinterpret_cast<FieldStats *>(partials);
    dnsmc::note_launch();
    if (srcX) pack_stats_kernel<true><<<blocks, kStatThreads, 0, (cudaStream_t)stream>>>(srcT, srcX, dst, na, nb, n, si, sj, sk, base, part, out);
    else pack_stats_kernel<false><<<blocks, kStatThreads, 0, (cudaStream_t)stream>>>(srcT, srcX, dst, na, nb, n, si, sj, sk, base, part, out);
    return (int)cudaGetLastError();
}
int launch_field_stats(int kind, const float *v, long long n, double *partials, double *out, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    dnsmc::note_launch();
    FieldStats *part = reinterpret_cast<FieldStats *>(partials);
    if (kind == STATS_T) field_stats_kernel<STATS_T><<<kStatBlocks, kStatThreads, 0, st>>>(v, n, part, out);
    else if (kind == STATS_TX) field_stats_kernel<STATS_TX><<<kStatBlocks, kStatThreads, 0, st>>>(v, n, part, out);
    else field_stats_kernel<STATS_V><<<kStatBlocks, kStatThreads, 0, st>>>(v, n, part, out);
    return (int)cudaGetLastError();
}

int field_stats_partials() { return 4 * kStatBlocks; }

int upload_sobol_dirs(const uint32_t dirs[4][32]) {
    int rc = (int)cudaMemcpyToSymbol(c_sobol, dirs, sizeof(uint32_t) * 4 * 32);
    if (rc) return rc;
    rc = upload_sobol_dirs_gen(dirs);
    return rc ? rc : upload_sobol_dirs_pair(dirs);
}

int device_sm_count() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    return n;
}

}  // namespace dnsmc
