// mc_ckgen.cu -- correlated-k tables from line-by-line absorption spectra on
// the GPU: the reference's offline generator (distr/correlatedK.cpp:145-300,
// correlatedKT; the band means of distr/calc_prob.cpp:17-119), for every
// (temperature, H2O mole fraction, narrow band) at once.
//
// Per band of one spectrum (one CTA of 256 threads):
//   kmin, kmax over the band's points;
//   n_pwrk bins uniform in k^0.1 between kmin^0.1 and kmax^0.1; every
//   interval h of the band's points (midpoint k of points h-1 and h) lands
//   in bin 1 + floor((k^0.1 - kmin^0.1) / step) -- the reference's
//   MAX(0, (int)((kpwri - pwrk_min) / pwrk_step + 1)) -- counted in shared
//   memory;
//   the g-function g(h) = 1 - sum over bins b = h+1 .. n_pwrk-1 of the
//   spectral fraction of bin b, the fraction being count * dwv / band width
//   (the spectrum is uniform in wavenumber; the reference sums dwv / width
//   point by point, the same value up to rounding);
//   bin values k(h) = (e(h) + e(h+1)) / 2 with e(h) = (kmin^0.1 + h step)^10
//   (ten-fold products, not a power function: the host oracle gives the
//   same bits);
//   k at every quadrature point g_r by linear interpolation in g between
//   the bins that bracket it (the first h with g(h+1) >= g_r);
//   the band mean of k, sum over bins 1 .. n_pwrk-1 of k(h) x fraction(h)
//   (calc_prob.cpp's k_avg), in a fixed order.
//
// What bounds it is FP64, which this GPU does at 2 per clock and SM: a power
// per point and 18 operations per filled bin.  A point's bin is therefore
// found in FP32 first, with an error bound; only where the bound reaches a bin
// edge is k^0.1 refined in FP64 (a Newton step from the FP32 value, good to
// 1e-12), and only where that is still undecided (bin position within 1e-6
// of an edge) is the power itself taken, so every count is the one the FP64
// power gives.  52 spectra x 32 bands of 2500 points, 10000 bins: 5.65 ms (a power
// a point, the mean by one thread), now 0.33 ms.
// Compiled with -fmad=false like the marches: the oracle (oracle/mc_oracle.cpp,
// orc_ck_from_lbl, built with -ffp-contract=off) reproduces every value up
// to the power k^0.1 of the bin boundaries.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/dnsmc.h"
#include "mc_internal.h"

namespace dnsmc {

int report_error(int code, const char *msg);  // mc_host.cpp

namespace {

constexpr int kCkThreads = 256;

struct CkGenParams {
    const double *kappa;      // [nT][nX][npts]
    long long npts;
    long long item0;          // the launch's first item
    int nT, nX, nbands, nq, n_pwrk;
    const long long *first;   // [nbands]
    const int *count;         // [nbands]
    const double *frac;       // [nbands] dwv / (wv_right - wv_left)
    const double *gq;         // [nq]
    float *kq;                // [nbands][nq][nT][nX]
    double *kavg;             // [nT][nX][nbands] or null
};

// (p0 + h * step)^10 as products
__device__ __forceinline__ double ck_edge(double p0, double step, int h) {
    const double x = (double)h * step + p0;
    const double x2 = x * x;
    const double x4 = x2 * x2;
    const double x5 = x4 * x;
    return x5 * x5;
}

__device__ __forceinline__ double ck_bin_k(double p0, double step, int h) {
    return 0.5 * (ck_edge(p0, step, h) + ck_edge(p0, step, h + 1));
}

// Bin of the interval between two neighbouring points of k: the value of
//   min(max((int)((pow((a + b) / 2, 0.1) - p0) / step + 1.0), 0), NB).
__device__ __forceinline__ int ck_bin(double a, double b, double p0, double step, float p0f, float invf, int NB) {
    const float kf = 0.5f * ((float)a + (float)b);
    if (kf > 1e-30f && kf < 1e30f) {
        // k^0.1 = 2^q 2^(r/10) 2^(log2(m)/10), k = 2^(10 q + r) m, m in
        // [0.75, 1.5): the three factors and their product are good to
        // 2.5e-7 relative (log2f and exp2f to 2 ulp)
        const uint32_t u = __float_as_uint(kf) - 0x3f400000u;       // bits relative to 0.75
        const int e = (int)u >> 23;                                   // 10 q + r
        const float m = __uint_as_float((u & 0x7fffffu) + 0x3f400000u);
        const int q = (e + 1000) / 10 - 100, r = e - 10 * q;
        const float y = ldexpf(exp2f(0.1f * (float)r) * exp2f(0.1f * log2f(m)), q);
        // its bin position, and how far that can be off: the 2.5e-7 and
        // exp2f(r/10)'s 2.5e-7 of y, p0's rounding, three FP32 roundings of t
        const float t = fmaf(y - p0f, invf, 1.0f);
        const float err = fmaf(6e-7f, fmaf(y, invf, p0f * invf), 3e-7f * fabsf(t)) + 1e-6f;
        const float f = t - floorf(t);
        if (f > err && f < 1.0f - err) return min(max((int)t, 0), NB);
        // near an edge: one Newton step for y^10 = k in FP64 (4.5 times the
        // square of y's error: below 2e-12 relative), its reciprocal in FP32
        const double k = (a + b) / 2.0, yd = (double)y;
        const double y2 = yd * yd, y4 = y2 * y2, y10 = y4 * y4 * y2;
        const double y1 = yd + yd * ((k - y10) * (double)(0.1f / (float)y10));
        const double td = (y1 - p0) * (double)invf + 1.0;
        // off by invf's rounding, the Newton step's error and FP64's in y1 and p0
        const double fl = floor(td), fd = td - fl, ed = 1e-7 * fabs(td) + 1e-11 * (y1 + p0) * (double)invf + 1e-6;
        if (fd > ed && fd < 1.0 - ed) return min(max((int)fl, 0), NB);
    }
    const double ki = (a + b) / 2.0;
    return min(max((int)((pow(ki, 0.1) - p0) / step + 1.0), 0), NB);
}

__global__ void __launch_bounds__(kCkThreads) ck_distribution_kernel(const CkGenParams P) {
    extern __shared__ unsigned int s_cnt[];   // n_pwrk + 2 counts, then suffix sums
    __shared__ long long s_red[2][kCkThreads / 32];
    __shared__ unsigned int s_part[kCkThreads / 32];
    __shared__ double s_sum[kCkThreads / 32], s_bins[3];
    __shared__ int s_queue[kCkThreads / 32][64];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long item = P.item0 + blockIdx.x;  // (t * nX + x) * nbands + band
    const int band = (int)(item % P.nbands);
    const long long tx = item / P.nbands;
    const double *kv = P.kappa + tx * P.npts + P.first[band];
    const int n = P.count[band];
    const int NB = P.n_pwrk;

    // kmin, kmax over the band's points (as integers: the order of
    // non-negative doubles)
    long long blo = 0x7fffffffffffffffLL, bhi = -0x7fffffffffffffffLL - 1;
    for (int h = tid; h < n; h += kCkThreads) {
        const long long v = __double_as_longlong(kv[h]);
        blo = min(blo, v);
        bhi = max(bhi, v);
    }
    for (int o = 16; o > 0; o >>= 1) {
        blo = min(blo, __shfl_xor_sync(0xffffffffu, blo, o));
        bhi = max(bhi, __shfl_xor_sync(0xffffffffu, bhi, o));
    }
    if (lane == 0) { s_red[0][warp] = blo; s_red[1][warp] = bhi; }
    for (int b = tid; b < NB + 2; b += kCkThreads) s_cnt[b] = 0u;
    __syncthreads();
    blo = s_red[0][0];
    bhi = s_red[1][0];
    for (int w = 1; w < kCkThreads / 32; ++w) { blo = min(blo, s_red[0][w]); bhi = max(bhi, s_red[1][w]); }
    const double lo = __longlong_as_double(blo), hi = __longlong_as_double(bhi);
    const int t_ = (int)(tx / P.nX), x_ = (int)(tx % P.nX);
    const long long TX = (long long)P.nT * P.nX;
    if (!(hi > lo)) {  // a flat band: k is the same at every g
        if (tid < P.nq) P.kq[((long long)band * P.nq + tid) * TX + t_ * P.nX + x_] = (float)lo;
        if (tid == 0 && P.kavg) P.kavg[tx * P.nbands + band] = lo;
        return;
    }
    // (one warp: every warp's copy would cost as much FP64 as its points)
    if (warp == 0) {
        const double pw = pow(lane ? hi : lo, 0.1);
        const double q0 = __shfl_sync(0xffffffffu, pw, 0), q1 = __shfl_sync(0xffffffffu, pw, 1);
        const double st = (q1 - q0) / (double)(NB - 1);
        if (lane == 0) { s_bins[0] = q0; s_bins[1] = st; s_bins[2] = 1.0 / st; }
    }
    __syncthreads();
    const double p0 = s_bins[0], step = s_bins[1];
    // bins of the intervals between neighbouring points
    const float p0f = (float)p0, invf = (float)s_bins[2];
    for (int h = 1 + tid; h < n; h += kCkThreads) atomicAdd(&s_cnt[ck_bin(kv[h], kv[h - 1], p0, step, p0f, invf, NB)], 1u);
    __syncthreads();
    // suffix sums over bins 1 .. NB-1 (the bins the g-function uses):
    // s_cnt[h] <- sum_{b = h .. NB-1} count[b] for h = 1 .. NB, 0 at NB; a run
    // of bins a thread (odd, so that the threads' runs start on other banks)
    const int per = ((NB + kCkThreads - 1) / kCkThreads) | 1;
    const int b0 = min(NB, 1 + tid * per), b1 = min(NB, b0 + per);
    {
        unsigned int acc = 0;
        for (int b = b0; b < b1; ++b) acc += s_cnt[b];
        unsigned int suf = acc;  // this thread's and the later threads' of the warp
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int v = __shfl_down_sync(0xffffffffu, suf, o);
            if (lane + o < 32) suf += v;
        }
        if (lane == 0) s_part[warp] = suf;
        __syncthreads();
        unsigned int run = suf - acc;  // bins after this thread's run
        for (int q = warp + 1; q < kCkThreads / 32; ++q) run += s_part[q];
        for (int b = b1 - 1; b >= b0; --b) {
            run += s_cnt[b];
            s_cnt[b] = run;
        }
        if (tid == 0) s_cnt[NB] = 0u;
        __syncthreads();
    }
    const double frac = P.frac[band];
    // g(h) = 1 - (suffix count from h + 1) x frac, h = 0 .. NB-1
    auto g_at = [&](int h) -> double { return 1.0 - (double)s_cnt[h + 1] * frac; };
    if (tid < P.nq) {
        const double g = P.gq[tid];
        // first t in [0, NB-2] with g(t+1) >= g (g(NB-1) = 1 >= g)
        int a = 0, z = NB - 2;
        while (a < z) {
            const int m = (a + z) >> 1;
            if (g_at(m + 1) >= g) z = m; else a = m + 1;
        }
        const int t = a;
        const double g0 = g_at(t), g1 = g_at(t + 1);
        const double k0 = ck_bin_k(p0, step, t), k1 = ck_bin_k(p0, step, t + 1);
        const double kq = (g1 == g0) ? k1 : k0 + (k1 - k0) * (g - g0) / (g1 - g0);
        P.kq[((long long)band * P.nq + tid) * TX + t_ * P.nX + x_] = (float)kq;
    }
    if (P.kavg) {
        // an eighth of the bins a warp; the filled ones (a quarter, typically)
        // are queued so that 32 of them share the FP64 instructions
        double s = 0.0;
        auto add = [&](int h) { s += ck_bin_k(p0, step, h) * ((double)(s_cnt[h] - s_cnt[h + 1]) * frac); };
        const int wper = (NB + kCkThreads / 32 - 1) / (kCkThreads / 32);
        const int h0 = 1 + warp * wper, h1 = min(NB, h0 + wper);
        int *const q = s_queue[warp];
        int nq = 0;
        for (int hb = h0; hb < h1; hb += 32) {
            const int h = hb + lane;
            const bool on = h < h1 && s_cnt[h] != s_cnt[h + 1];
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) q[nq + __popc(m & ((1u << lane) - 1u))] = h;
            nq += __popc(m);
            __syncwarp();
            if (nq >= 32) {
                add(q[lane]);
                const int v = q[32 + lane];
                __syncwarp();
                q[lane] = v;
                nq -= 32;
                __syncwarp();
            }
        }
        if (lane < nq) add(q[lane]);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) s_sum[warp] = s;
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < kCkThreads / 32; ++w) s += s_sum[w];
            P.kavg[tx * P.nbands + band] = s;
        }
    }
}

// Whether every value is finite and >= 0 (-0 among them), on the bits.
__global__ void ck_check_kernel(const double *k, long long n, unsigned int *bad) {
    unsigned int b = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long v = (unsigned long long)__double_as_longlong(k[i]);
        b |= v >= 0x7ff0000000000000ull && v != 0x8000000000000000ull ? 1u : 0u;
    }
    if (__any_sync(0xffffffffu, b) && (threadIdx.x & 31) == 0) atomicOr(bad, 1u);
}

template <class T>
struct Dev {
    T *p = nullptr;
    ~Dev() { if (p) cudaFree(p); }
    cudaError_t alloc(size_t n) { return cudaMalloc((void **)&p, (n ? n : 1) * sizeof(T)); }
};

// Streams of one call, idle when it returns.
struct Streams {
    static constexpr int kMax = 4;
    cudaStream_t s[kMax] = {};
    ~Streams() { for (cudaStream_t t : s) if (t) { cudaStreamSynchronize(t); cudaStreamDestroy(t); } }
};

}  // namespace
}  // namespace dnsmc

using namespace dnsmc;

extern "C" int dnsmc_ck_from_lbl(const dnsmc_lbl_desc *d, float *kq, double *kavg) {
    if (!d || !kq || !d->kappa || !d->first || !d->count || !d->wv_left || !d->wv_right || !d->gq)
        return report_error(DNSMC_ERR_ARG, "null argument");
    if (d->nT < 1 || d->nX < 1 || d->npts < 2 || d->nbands < 1 || d->nq < 1 || d->n_pwrk < 2)
        return report_error(DNSMC_ERR_ARG, "sizes must be >= 1 (npts, n_pwrk >= 2)");
    if (!(d->dwv > 0)) return report_error(DNSMC_ERR_ARG, "dwv must be > 0");
    // the bin counts live in shared memory
    if (d->n_pwrk > 50000) return report_error(DNSMC_ERR_ARG, "n_pwrk must be <= 50000");
    std::vector<double> frac((size_t)d->nbands);
    for (int b = 0; b < d->nbands; ++b) {
        if (d->count[b] < 2 || d->first[b] < 0 || d->first[b] + d->count[b] > d->npts)
            return report_error(DNSMC_ERR_ARG, "every band needs >= 2 points inside the spectrum");
        const double w = d->wv_right[b] - d->wv_left[b];
        if (!(w > 0)) return report_error(DNSMC_ERR_ARG, "band edges must satisfy wv_left < wv_right");
        frac[(size_t)b] = d->dwv / w;
    }
    for (int r = 0; r < d->nq; ++r)
        if (!(d->gq[r] > 0) || !(d->gq[r] < 1) || (r && !(d->gq[r] > d->gq[r - 1])))
            return report_error(DNSMC_ERR_ARG, "quadrature points must ascend inside (0, 1)");
    const long long nk = (long long)d->nT * d->nX * d->npts;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) {
        // (bad spectra are reported before a missing device; with one, the
        // device looks them over)
        for (long long i = 0; i < nk; ++i)
            if (!(d->kappa[i] >= 0) || !std::isfinite(d->kappa[i]))
                return report_error(DNSMC_ERR_TABLE, "absorption spectra must be finite and >= 0");
        return report_error(DNSMC_ERR_NODEVICE, "no CUDA device");
    }
    const long long items = (long long)d->nT * d->nX * d->nbands;
    if (items > 0x7fffffffLL) return report_error(DNSMC_ERR_ARG, "too many (T, x, band) items");
    // one allocation: spectra | small inputs (frac, gq, first, count, flag) | kavg | kq
    const size_t B = (size_t)d->nbands;
    const size_t o_frac = 0, o_gq = o_frac + B * 8, o_first = o_gq + (size_t)d->nq * 8, o_count = o_first + B * 8,
                 o_bad = o_count + (B + 1) / 2 * 8, n_small = o_bad + 8;
    const size_t a_kavg = ((size_t)nk * 8 + n_small + 255) / 256 * 256, a_kq = a_kavg + (size_t)items * 8;
    std::vector<unsigned char> small(n_small, 0);
    memcpy(small.data() + o_frac, frac.data(), B * 8);
    memcpy(small.data() + o_gq, d->gq, (size_t)d->nq * 8);
    memcpy(small.data() + o_first, d->first, B * 8);
    memcpy(small.data() + o_count, d->count, B * 4);
    Dev<unsigned char> mem;
    cudaError_t e = mem.alloc(a_kq + (size_t)items * d->nq * 4);
    if (e != cudaSuccess) return report_error(DNSMC_ERR_NOMEM, cudaGetErrorString(e));
    unsigned char *in = mem.p + (size_t)nk * 8;
    // (the copy of pageable memory may still be under way when cudaMemcpy
    // returns, and the streams below do not wait for the default stream)
    e = cudaMemcpy(in, small.data(), n_small, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);
    if (e != cudaSuccess) return report_error(DNSMC_ERR_CUDA, cudaGetErrorString(e));
    unsigned int *bad = (unsigned int *)(in + o_bad);
    CkGenParams P{};
    P.kappa = (const double *)mem.p; P.npts = d->npts; P.nT = d->nT; P.nX = d->nX; P.nbands = d->nbands; P.nq = d->nq;
    P.n_pwrk = d->n_pwrk; P.first = (const long long *)(in + o_first); P.count = (const int *)(in + o_count);
    P.frac = (const double *)(in + o_frac); P.gq = (const double *)(in + o_gq);
    P.kq = (float *)(mem.p + a_kq); P.kavg = kavg ? (double *)(mem.p + a_kavg) : nullptr;
    const size_t smem = (size_t)(d->n_pwrk + 2) * sizeof(unsigned int);
    if (smem > 48 * 1024) {
        e = cudaFuncSetAttribute(ck_distribution_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return report_error(DNSMC_ERR_ARG, "n_pwrk too large for shared memory");
    }
    // Spectra of 8 MB and more go over in four parts, each with its own stream,
    // so that a part's kernels run while the next is copied.  52 spectra of 80001
    // points (33 MB): 760 -> 690 us (2 parts 745, 8 parts 740).
    const long long ntx = (long long)d->nT * d->nX;
    const int parts = nk * 8 >= (8 << 20) ? (int)std::min<long long>(Streams::kMax, ntx) : 1;
    Streams st;
    for (int c = 0; c < parts && e == cudaSuccess; ++c) {
        const long long t0 = ntx * c / parts, t1 = ntx * (c + 1) / parts;
        const double *kc = P.kappa + t0 * d->npts;
        const long long n = (t1 - t0) * d->npts;
        e = cudaStreamCreateWithFlags(&st.s[c], cudaStreamNonBlocking);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync((void *)kc, d->kappa + t0 * d->npts, (size_t)n * sizeof(double), cudaMemcpyHostToDevice, st.s[c]);
        if (e != cudaSuccess) break;
        dnsmc::note_launch();
        ck_check_kernel<<<(unsigned)std::min<long long>(608, (n + 255) / 256), 256, 0, st.s[c]>>>(kc, n, bad);
        P.item0 = t0 * d->nbands;
        dnsmc::note_launch();
        ck_distribution_kernel<<<(unsigned)((t1 - t0) * d->nbands), kCkThreads, smem, st.s[c]>>>(P);
        e = cudaGetLastError();
    }
    for (int c = 0; c < parts && e == cudaSuccess; ++c) e = cudaStreamSynchronize(st.s[c]);
    unsigned int hbad = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&hbad, bad, sizeof hbad, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return report_error(DNSMC_ERR_CUDA, cudaGetErrorString(e));
    if (hbad) return report_error(DNSMC_ERR_TABLE, "absorption spectra must be finite and >= 0");
    e = cudaMemcpy(kq, P.kq, (size_t)items * d->nq * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && kavg) e = cudaMemcpy(kavg, P.kavg, (size_t)items * sizeof(double), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return report_error(DNSMC_ERR_CUDA, cudaGetErrorString(e));
    return DNSMC_OK;
}
