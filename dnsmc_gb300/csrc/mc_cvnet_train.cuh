// mc_cvnet_train.cuh -- one training step of the network on the fifth-generation
// tensor cores, in three launches.  Included by mc_cvnet.cu after
// mc_cvnet_tc.cuh (descriptors, MMA, waits, tensor-memory loads).
//
//   train_tile_kernel   a 128-row tile per CTA through forward, loss and the
//                       input gradients without leaving the SM: the three
//                       hidden pre-activations stay in tensor memory (384 of
//                       its 512 columns), the weights and their transposes in
//                       shared memory; activations and dZ go out as bf16;
//   train_wgrad_kernel  dW = dZ^T H of all four layers, split over the rows;
//   train_update_kernel sums of the splits in a fixed order, column sums for
//                       the biases, Adam, the bf16 weight copies.
//
// A batch of 4096 rows is only 32 tiles, so a step is latency: what bounds it
// are the chain of seven layers with their epilogues and the launches.  Sixteen
// warps share a tile's epilogue (each 32 rows x 32 columns).  Per step of 4096
// rows: 478 us in 19 launches (a GEMM per layer and direction with 2-byte
// operand loads, one warpgroup per tile), now 58 us (32 + 16 + 10).
#pragma once

namespace {

constexpr int TR_THREADS = 512;
// transposed weight copies after the NWEIGHT elements of the forward ones:
// element (out, in) of W as B operand with N = in, K = out
constexpr long long WT_2 = NWEIGHT;
constexpr long long WT_3 = WT_2 + (long long)HID * HID;
constexpr long long WT_4 = WT_3 + (long long)HID * HID;
constexpr long long NWEIGHT_ALL = WT_4 + (long long)NOUT * HID;
// shared-memory map (bytes)
constexpr uint32_t TR_WT2 = TC_WBYTES;
constexpr uint32_t TR_WT3 = TR_WT2 + HID * HID * 2;
constexpr uint32_t TR_WT4 = TR_WT3 + HID * HID * 2;
constexpr uint32_t TR_WBYTES = TR_WT4 + NOUT * HID * 2;
constexpr uint32_t TR_BIAS = TR_WBYTES;
constexpr uint32_t TR_ACT = (TR_BIAS + (3 * HID + NOUT) * 4 + 127) / 128 * 128;
constexpr uint32_t TR_BAR = TR_ACT + TC_ACT_BYTES;
constexpr uint32_t TR_LOSS = TR_BAR + 32;
constexpr uint32_t TR_SMEM = TR_LOSS + 3 * (TR_THREADS / 32) * 8;
static_assert(TR_WBYTES == NWEIGHT_ALL * 2, "weight copy size");
static_assert(TR_SMEM <= 227 * 1024, "shared memory of the training tile");

struct TrainParams {
    long long rows, nvalid;   // rows of the batch (a multiple of 128), real ones
    const bf16 *X;            // [*][K0]
    const float *lab;         // [*][G][NLAB]
    const int *idx;           // row r is row idx[r] of X and lab (null: r)
    int G;
    float Sbeta, Sv, Sc, ridge;
    const bf16 *W;            // NWEIGHT_ALL: tensor-core order, then the transposes
    const float *P;           // FP32 master parameters (biases)
    bf16 *H0, *H1, *H2, *H3;  // [rows][K0], [rows][HID]
    bf16 *dO, *dZ3, *dZ2, *dZ1;  // [rows][NOUT], [rows][HID]
    double *part;             // [tile][3]: beta, variance, cost loss sums
    unsigned int *status;
};

// 16 consecutive f32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 bf16 columns of this thread's row (chunks 4 cg .. 4 cg + 3) to the A tile
// and to the row in memory
__device__ __forceinline__ void train_store32(unsigned char *act, int row, int cg, const uint32_t (&h)[16], bf16 *dst) {
    uint4 *d = reinterpret_cast<uint4 *>(dst + cg * 32);
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const uint4 u = make_uint4(h[4 * m], h[4 * m + 1], h[4 * m + 2], h[4 * m + 3]);
        *reinterpret_cast<uint4 *>(act + (cg * 4 + m) * (TC_TILE * 16) + row * 16) = u;
        d[m] = u;
    }
}

// Loss: per row and band-group slot g < G
//   beta loss  (V(beta) + ridge (Caa da^2 + Cbb db^2)) / S_beta
//   var loss   (v / S_v) exp(-o_v) + o_v     (minimiser: o_v = log E[v / S_v])
//   cost loss  (c / S_c) exp(-o_c) + o_c
// mean over rows; d = d(mean)/d out of the slot's four outputs.
__device__ __forceinline__ void train_loss(const TrainParams &L, const float *y, const float *o, float inv, float *d,
                                           double &lb, double &lv, double &lc) {
    const float Cxx = y[0], Caa = y[1], Cbb = y[2], Cxa = y[3], Cxb = y[4], Cab = y[5];
    const float da = o[0], db = o[1];
    const float ba = 1.0f + da, bb = -1.0f + db;
    const float V = Cxx - 2.0f * ba * Cxa - 2.0f * bb * Cxb + ba * ba * Caa + 2.0f * ba * bb * Cab + bb * bb * Cbb;
    lb += (double)((V + L.ridge * (Caa * da * da + Cbb * db * db)) / L.Sbeta);
    // (contractions written out: the same rounding wherever this is inlined)
    d[0] = fmaf(2.0f * L.ridge * Caa, da, 2.0f * (fmaf(ba, Caa, bb * Cab) - Cxa)) / L.Sbeta * inv;
    d[1] = fmaf(2.0f * L.ridge * Cbb, db, 2.0f * (fmaf(ba, Cab, bb * Cbb) - Cxb)) / L.Sbeta * inv;
    if (y[6] > 0.0f) {
        const float ov = clampo(o[2]), v = y[6] / L.Sv, ex = expf(-ov);
        lv += (double)fmaf(v, ex, ov);
        d[2] = fmaf(-v, ex, 1.0f) * inv;
    }
    if (y[7] > 0.0f) {
        const float oc = clampo(o[3]), c = y[7] / L.Sc, ex = expf(-oc);
        lc += (double)fmaf(c, ex, oc);
        d[3] = fmaf(-c, ex, 1.0f) * inv;
    }
}

// The three kernels of a step follow one another with programmatic dependence
// (launch_step): each lets the next one's blocks be placed as soon as its own
// have started, and waits for the one before to have finished before it
// touches memory.
__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__global__ void __launch_bounds__(TR_THREADS, 1) train_tile_kernel(const TrainParams F) {
    step_begin();
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, cg = warp >> 2;  // this thread's tile row and column group
    uint64_t *bar_w = reinterpret_cast<uint64_t *>(sm + TR_BAR), *bar_m = bar_w + 1;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + TR_BAR + 16);
    float *bias = reinterpret_cast<float *>(sm + TR_BIAS);
    double *s_loss = reinterpret_cast<double *>(sm + TR_LOSS);
    unsigned char *act = sm + TR_ACT;
    const uint32_t act_a = tc_smem(act), w_a = tc_smem(sm);
    unsigned int err = 0;

    if (tid == 0) {
        for (int b = 0; b < 2; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(bar_w + b)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int e = tid; e < 3 * HID + NOUT; e += TR_THREADS)
        bias[e] = F.P[e < HID ? OFF_B1 + e : (e < 2 * HID ? OFF_B2 + e - HID : (e < 3 * HID ? OFF_B3 + e - 2 * HID : OFF_B4 + e - 3 * HID))];
    if (warp == 0) {  // Z1, Z2, Z3 at columns 0, 128, 256; the accumulator of the output layer and the gradients at 384
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tc_smem(tslot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    if (tid == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(bar_w)), "r"(TR_WBYTES) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(w_a),
                     "l"(F.W), "r"(TR_WBYTES), "r"(tc_smem(bar_w))
                     : "memory");
    }
    const float inv = 1.0f / (float)max(1LL, F.nvalid);
    uint32_t ph = 0;
    bool loaded = false;
    // the A tile is complete: one elected thread issues the layer's MMAs into
    // the 128 columns at `col`, every thread waits for them
    auto layer = [&](int which, uint32_t col) {
        tc_proxy_fence();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t d = tmem + col;
            if (which == 0) tc_layer<K0, HID>(act_a, w_a + TC_W1, d, bar_m);
            else if (which == 1) tc_layer<HID, HID>(act_a, w_a + TC_W2, d, bar_m);
            else if (which == 2) tc_layer<HID, HID>(act_a, w_a + TC_W3, d, bar_m);
            else if (which == 3) tc_layer<HID, NOUT>(act_a, w_a + TC_W4, d, bar_m);
            else if (which == 4) tc_layer<NOUT, HID>(act_a, w_a + TR_WT4, d, bar_m);
            else if (which == 5) tc_layer<HID, HID>(act_a, w_a + TR_WT3, d, bar_m);
            else tc_layer<HID, HID>(act_a, w_a + TR_WT2, d, bar_m);
        }
        if (!tc_wait(bar_m, ph)) err |= DNSMC_STATUS_COPY_TIMEOUT;
        ph ^= 1u;
        tc_fence_after();
    };
    const long long ntiles = F.rows / TC_TILE;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long r = tile * TC_TILE + row;
        const bool valid = r < F.nvalid;
        const long long sr = valid && F.idx ? (long long)F.idx[r] : r;
        // ---- layer-1 input
        for (int c = cg; c < K0 / 8; c += 4) {
            const uint4 u = valid ? *reinterpret_cast<const uint4 *>(F.X + sr * K0 + c * 8) : make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4 *>(act + c * (TC_TILE * 16) + row * 16) = u;
            *reinterpret_cast<uint4 *>(F.H0 + r * K0 + c * 8) = u;
        }
        if (!loaded) {
            if (!tc_wait(bar_w, 0)) err |= DNSMC_STATUS_COPY_TIMEOUT;
            loaded = true;
        }
        // ---- hidden layers: Z stays in tensor memory
#pragma unroll 1
        for (int l = 0; l < 3; ++l) {
            layer(l, (uint32_t)l * HID);
            uint32_t v[32], h[16];
            tc_ld32(tlane + l * HID + cg * 32, v);
            const float *b = bias + l * HID + cg * 32;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                h[q] = pack_bf16(gelu(__uint_as_float(v[2 * q]) + b[2 * q]), gelu(__uint_as_float(v[2 * q + 1]) + b[2 * q + 1]));
            train_store32(act, row, cg, h, (l == 0 ? F.H1 : (l == 1 ? F.H2 : F.H3)) + r * HID);
        }
        // ---- output layer and loss: four band-group slots of this row
        layer(3, 3 * HID);
        double lb = 0.0, lv = 0.0, lc = 0.0;
        {
            uint32_t v[16];
            tc_ld16(tlane + 3 * HID + cg * 16, v);
            float d[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) d[q] = 0.0f;
            if (valid) {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int g = cg * 4 + s;
                    if (g >= F.G) break;
                    float o[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) o[q] = __uint_as_float(v[4 * s + q]) + bias[3 * HID + 4 * g + q];
                    const float4 *y = reinterpret_cast<const float4 *>(F.lab + (sr * F.G + g) * NLAB);
                    const float4 y0 = y[0], y1 = y[1];
                    const float yy[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
                    train_loss(F, yy, o, inv, d + 4 * s, lb, lv, lc);
                }
            }
            uint4 *dst = reinterpret_cast<uint4 *>(F.dO + r * NOUT + cg * 16);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                const uint4 u = make_uint4(pack_bf16(d[8 * m], d[8 * m + 1]), pack_bf16(d[8 * m + 2], d[8 * m + 3]),
                                           pack_bf16(d[8 * m + 4], d[8 * m + 5]), pack_bf16(d[8 * m + 6], d[8 * m + 7]));
                *reinterpret_cast<uint4 *>(act + (cg * 2 + m) * (TC_TILE * 16) + row * 16) = u;
                dst[m] = u;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lb += __shfl_xor_sync(0xffffffffu, lb, o);
            lv += __shfl_xor_sync(0xffffffffu, lv, o);
            lc += __shfl_xor_sync(0xffffffffu, lc, o);
        }
        if (lane == 0) { s_loss[warp * 3] = lb; s_loss[warp * 3 + 1] = lv; s_loss[warp * 3 + 2] = lc; }
        // ---- input gradients: dZ_l = (dZ_{l+1} W) GELU'(Z_l)
#pragma unroll 1
        for (int l = 2; l >= 0; --l) {
            layer(6 - l, 3 * HID);
            if (l == 2 && tid < 3) {  // (the layer's barrier is behind s_loss)
                double t = 0.0;
                for (int w = 0; w < TR_THREADS / 32; ++w) t += s_loss[w * 3 + tid];
                F.part[tile * 3 + tid] = t;
            }
            uint32_t a[32], z[32], h[16];
            tc_ld32(tlane + 3 * HID + cg * 32, a);
            tc_ld32(tlane + l * HID + cg * 32, z);
            const float *b = bias + l * HID + cg * 32;
#pragma unroll
            for (int q = 0; q < 16; ++q)
                h[q] = pack_bf16(__uint_as_float(a[2 * q]) * gelu_grad(__uint_as_float(z[2 * q]) + b[2 * q]),
                                 __uint_as_float(a[2 * q + 1]) * gelu_grad(__uint_as_float(z[2 * q + 1]) + b[2 * q + 1]));
            train_store32(act, row, cg, h, (l == 2 ? F.dZ3 : (l == 1 ? F.dZ2 : F.dZ1)) + r * HID);
        }
        tc_fence_before();
        __syncthreads();  // the next tile overwrites the A tile, s_loss and the accumulators
        tc_fence_after();
    }
    if (err && F.status) atomicOr(F.status, err);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Weight gradients: blockIdx.y the layer, blockIdx.x the split of klen rows.
// The MMA's K runs over the batch rows, so both operands are transposed on
// their way to shared memory: a warp reads 8 rows x 32 columns (16 bytes a
// lane) and stores 2-byte elements; the lanes of a row start at different
// columns, which keeps the four groups of 8 lanes off each other's banks.
// 256 rows at a time, 16 MMAs of K 16, f32 accumulators in tensor memory.
// ---------------------------------------------------------------------------
constexpr int WG_K = 256, WG_THREADS = 256;
constexpr int WG_SMEM = 2 * WG_K * 128 * 2;  // 128 KB: one CTA per SM

struct WgradParams {
    long long rows;
    int klen, splits;
    const bf16 *dZ[4], *H[4];  // layers 1 .. 4
    float *part;               // layer l at wg_part(l, splits): [split][out][in]
};

__host__ __device__ constexpr int wg_nout(int l) { return l == 3 ? NOUT : HID; }
__host__ __device__ constexpr int wg_nin(int l) { return l == 0 ? K0 : HID; }
__host__ __device__ constexpr long long wg_part(int l, int splits) {
    return (long long)splits * (l == 0 ? 0 : (l == 1 ? HID * K0 : (l == 2 ? HID * K0 + HID * HID : HID * K0 + 2 * HID * HID)));
}

// columns [0, ncol) of rows [k0, k0 + WG_K) of a row-major bf16 matrix into
// the K-major operand of `nrow` rows (zeros for the columns beyond ncol and the
// rows from kend on)
__device__ __forceinline__ void wg_stage(unsigned char *s, int nrow, const bf16 *src, int ncol, long long k0, long long kend) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kr = lane & 7, cc = lane >> 3;
    const int groups = (nrow + 31) / 32;  // of 32 columns
    const int n = (WG_K / 8) * groups;
    constexpr int B = 8;                  // loads in flight a lane
    for (int it0 = warp; it0 < n; it0 += B * (WG_THREADS / 32)) {
        uint4 u[B];
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int it = it0 + b * (WG_THREADS / 32);
            const int c0 = (it % groups) * 32 + cc * 8;
            const long long k = k0 + (it / groups) * 8 + kr;
            u[b] = it < n && k < kend && c0 < ncol ? *reinterpret_cast<const uint4 *>(src + k * ncol + c0)
                                                   : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) {
            const int it = it0 + b * (WG_THREADS / 32);
            const int kc = it / groups, c0 = (it % groups) * 32 + cc * 8;
            if (it >= n || c0 >= nrow) continue;
            const uint32_t w[4] = {u[b].x, u[b].y, u[b].z, u[b].w};
            unsigned char *d = s + kc * (nrow * 16) + c0 * 16 + kr * 2;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = (q + 2 * cc) & 7;
                const uint32_t v = j < 4 ? (j < 2 ? w[0] : w[1]) : (j < 6 ? w[2] : w[3]);
                *reinterpret_cast<uint16_t *>(d + j * 16) = (uint16_t)(j & 1 ? v >> 16 : v & 0xffffu);
            }
        }
    }
}

__global__ void __launch_bounds__(WG_THREADS, 1) train_wgrad_kernel(const WgradParams G, unsigned int *status) {
    step_begin();
    extern __shared__ __align__(1024) unsigned char gsm[];
    __shared__ uint64_t bar;
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int l = blockIdx.y, nout = wg_nout(l), nin = wg_nin(l);
    unsigned char *sA = gsm, *sB = gsm + WG_K * 128 * 2;
    const long long kbeg = (long long)blockIdx.x * G.klen, kend = min(G.rows, kbeg + G.klen);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(tc_smem(&tslot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;
    const uint32_t aA = tc_smem(sA), aB = tc_smem(sB);
    uint32_t ph = 0;
    unsigned int err = 0;
    for (long long k0 = kbeg; k0 < kend; k0 += WG_K) {
        wg_stage(sA, 128, G.dZ[l], nout, k0, kend);
        wg_stage(sB, nin, G.H[l], nin, k0, kend);
        tc_proxy_fence();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const int nk = (int)((min(kend, k0 + WG_K) - k0 + 15) / 16);
            for (int k = 0; k < nk; ++k) {
                const uint64_t da = tc_desc(aA + k * 2 * (128 * 16), 128 * 16, 128);
                const uint64_t db = tc_desc(aB + k * 2 * (nin * 16), nin * 16, 128);
                tc_mma(tmem, da, db, tc_idesc(128, nin), (k0 > kbeg || k > 0) ? 1u : 0u);
            }
            tc_commit(&bar);
        }
        if (!tc_wait(&bar, ph)) err |= DNSMC_STATUS_COPY_TIMEOUT;
        ph ^= 1u;
        tc_fence_after();
    }
    const int m = (warp & 3) * 32 + lane;
    const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    float *out = G.part + wg_part(l, G.splits) + ((long long)blockIdx.x * nout + m) * nin;
    for (int c = warp >> 2; c < nin / 16; c += 2) {
        uint32_t v[16];
        tc_ld16(tlane + c * 16, v);
        if (m >= nout) continue;
        float4 *o = reinterpret_cast<float4 *>(out + c * 16);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            o[q] = kend > kbeg ? make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                             __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]))
                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (err && status) atomicOr(status, err);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
    }
}

// ---------------------------------------------------------------------------
// Gradients and Adam.  Blocks [0, WU_WBLOCKS): a weight a thread, its partials
// summed in split order.  Then a block per 8 bias columns: thread t sums rows
// t, t + 256, ... of the eight columns (one 16-byte load a row), then a tree
// over the threads.
// ---------------------------------------------------------------------------
constexpr int WU_THREADS = 256;
constexpr int WU_WBLOCKS = (int)((NWEIGHT + WU_THREADS - 1) / WU_THREADS);
constexpr int WU_BBLOCKS = (3 * HID + NOUT) / 8;

struct UpdateParams {
    const float *part;
    int splits;
    long long rows;
    const bf16 *dZ[4];
    float *grad;              // [NPARAM]
    int adam;                 // 0: gradients only
    float *p, *m, *v;
    bf16 *w;                  // the bf16 weight copies
    float lr, b1, b2, eps, c1, c2;
};

__device__ __forceinline__ float adam_update(const UpdateParams &U, long long e, float gr) {
    // (the contraction written out: the same rounding wherever this is inlined)
    const float mm = fmaf(1.0f - U.b1, gr, U.b1 * U.m[e]);
    const float vv = fmaf((1.0f - U.b2) * gr, gr, U.b2 * U.v[e]);
    U.m[e] = mm;
    U.v[e] = vv;
    const float upd = U.lr * (mm / U.c1) / (sqrtf(vv / U.c2) + U.eps);
    const float p = U.p[e] - upd;
    U.p[e] = p;
    return p;
}

// the weight copies of element (out n, in k) of layer l: tensor-core order
// [in/8][out][8], and (layers 2 to 4) the transpose's [out/8][in][8]
__device__ __forceinline__ void store_weight(bf16 *w, int l, int n, int k, float v) {
    const long long off = l == 0 ? WOFF_1 : (l == 1 ? WOFF_2 : (l == 2 ? WOFF_3 : WOFF_4));
    const bf16 b = __float2bfloat16(v);
    w[off + tc_index(n, k, wg_nout(l))] = b;
    if (l) w[(l == 1 ? WT_2 : (l == 2 ? WT_3 : WT_4)) + tc_index(k, n, HID)] = b;
}

// weight number q (0 .. NWEIGHT - 1, row-major per layer): its layer, row,
// column and index in the parameters
__device__ __forceinline__ long long weight_at(long long q, int &l, int &n, int &k) {
    l = q < WOFF_2 ? 0 : (q < WOFF_3 ? 1 : (q < WOFF_4 ? 2 : 3));
    const long long e = q - (l == 0 ? WOFF_1 : (l == 1 ? WOFF_2 : (l == 2 ? WOFF_3 : WOFF_4)));
    n = (int)(e / wg_nin(l));
    k = (int)(e % wg_nin(l));
    return (l == 0 ? OFF_W1 : (l == 1 ? OFF_W2 : (l == 2 ? OFF_W3 : OFF_W4))) + e;
}

__global__ void __launch_bounds__(WU_THREADS) train_update_kernel(const UpdateParams U) {
    step_begin();
    if (blockIdx.x < WU_WBLOCKS) {
        const long long q = (long long)blockIdx.x * WU_THREADS + threadIdx.x;
        if (q >= NWEIGHT) return;
        int l, n, k;
        const long long e = weight_at(q, l, n, k);
        const long long sz = (long long)wg_nout(l) * wg_nin(l);
        const float *p = U.part + wg_part(l, U.splits) + (long long)n * wg_nin(l) + k;
        float s = 0.0f;
        // (not __ldg: with programmatic dependence the partials are written
        // while this kernel's blocks are already there)
#pragma unroll 8
        for (int z = 0; z < U.splits; ++z) s += __ldcg(p + z * sz);
        U.grad[e] = s;
        if (U.adam) store_weight(U.w, l, n, k, adam_update(U, e, s));
        return;
    }
    __shared__ float red[8][WU_THREADS];
    const int c = ((int)blockIdx.x - WU_WBLOCKS) * 8;            // column in b1 b2 b3 b4
    const int l = c < HID ? 0 : (c < 2 * HID ? 1 : (c < 3 * HID ? 2 : 3));
    const int n0 = c - l * HID, ncol = wg_nout(l), t = threadIdx.x;
    float s[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) s[j] = 0.0f;
#pragma unroll 8
    for (long long r = t; r < U.rows; r += WU_THREADS) {
        const uint4 u = *reinterpret_cast<const uint4 *>(U.dZ[l] + r * ncol + n0);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) red[j][t] = s[j];
    __syncthreads();
    for (int w = WU_THREADS / 2; w > 0; w >>= 1) {
        for (int q = t; q < 8 * w; q += WU_THREADS) red[q / w][q % w] += red[q / w][q % w + w];
        __syncthreads();
    }
    if (t < 8) {
        const long long e = (l == 0 ? OFF_B1 : (l == 1 ? OFF_B2 : (l == 2 ? OFF_B3 : OFF_B4))) + n0 + t;
        U.grad[e] = red[t][0];
        if (U.adam) adam_update(U, e, red[t][0]);
    }
}

// The bf16 weight copies of the master parameters (initial or loaded ones).
__global__ void weights_to_bf16_kernel(const float *p, bf16 *w) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < NWEIGHT; q += (long long)gridDim.x * blockDim.x) {
        int l, n, k;
        const long long e = weight_at(q, l, n, k);
        store_weight(w, l, n, k, p[e]);
    }
}

}  // namespace
