// dedisperse.cu -- incoherent dedispersion of a filterbank into DM trials
// (accel_dedisperse_delays, accel_dedisperse): the step upstream of the
// search that produces its input time series.  The reference takes series
// that are already dedispersed (its README names dedispersion as the step
// before it); this is the direct method in its textbook form:
//
//   out[d][t] = sum over channels c, in order, of in[c][t + delay[d][c]]
//   delay[d][c] = floor(kDM * DM_d * (f_c^-2 - f_ref^-2) / tsamp + 1/2)
//
// with the dispersion constant kDM = 4.148808e3 s MHz^2 pc^-1 cm^3, f_c the
// frequency of channel c (f_top + c * chan_bw) and f_ref the highest channel
// frequency, so that every delay is >= 0.
//
// Layout: filterbank channel-major [nchan][nsamp] float32 (time contiguous),
// output [ndm][nout] float32 with nout <= nsamp - max delay.  One CTA owns
// kDdD DM trials x kDdThreads*kDdPer consecutive output samples (each
// thread kDdPer samples kDdThreads apart, so every load of a warp is one
// contiguous run) and accumulates in registers over the channels in order
// (rounded float adds: the same sums as the host restatement).  The grid
// runs the DM tiles of one time window fastest, so the CTAs that read the
// same window of every channel run together and find it in L2.  The
// windowed form below (k_dedisperse_win) replaces it wherever a tile's
// delays lie close enough together for shared-memory windows.
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <vector>

#include "../../include/accelsearch.h"
#include "accel_internal.h"
#include "async_copy.cuh"

namespace accel {

constexpr int kDdThreads = 256;
constexpr int kDdPer = 4;  // output samples per thread
constexpr int kDdD = 8;    // DM trials per CTA (a multiple of 4: int4 delay loads)
static_assert(kDdD % 4 == 0, "delays are loaded as int4");
constexpr double kDispConst = 4.148808e3;

__global__ void __launch_bounds__(kDdThreads) k_dedisperse(const float* __restrict__ in, int nchan, long long nsamp,
                                                           const int4* __restrict__ dtab, int ndm, int ndtile,
                                                           float* __restrict__ out, long long nout) {
    const long long bid = blockIdx.x;
    const int tile = (int)(bid % ndtile);
    const int d0 = tile * kDdD;
    const long long t0 = (bid / ndtile) * (long long)(kDdThreads * kDdPer) + threadIdx.x;
    const int nd = min(kDdD, ndm - d0);
    float acc[kDdD][kDdPer];
#pragma unroll
    for (int j = 0; j < kDdD; j++)
#pragma unroll
        for (int k = 0; k < kDdPer; k++) acc[j][k] = 0.f;
    // dtab row c: the delays of channel c for the tile's kDdD DM trials as
    // kDdD/4 int4 (padding trials have delay 0 and are not summed)
    constexpr int kQ = kDdD / 4;
    const int4* __restrict__ dt = dtab + (long long)kQ * tile;
    const long long dstride = (long long)kQ * ndtile;
#pragma unroll 4
    for (int c = 0; c < nchan; c++) {
        const float* __restrict__ row = in + (long long)c * nsamp;
        int dl[kDdD];
#pragma unroll
        for (int q = 0; q < kQ; q++) {
            const int4 v = __ldg(dt + c * dstride + q);
            dl[4 * q] = v.x;
            dl[4 * q + 1] = v.y;
            dl[4 * q + 2] = v.z;
            dl[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < kDdD; j++) {
            if (j < nd) {  // uniform over the CTA
#pragma unroll
                for (int k = 0; k < kDdPer; k++) {
                    const long long t = t0 + (long long)k * kDdThreads;
                    if (t < nout) acc[j][k] = __fadd_rn(acc[j][k], __ldg(row + t + dl[j]));
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < kDdD; j++) {
        if (j < nd) {
#pragma unroll
            for (int k = 0; k < kDdPer; k++) {
                const long long t = t0 + (long long)k * kDdThreads;
                if (t < nout) out[(long long)(d0 + j) * nout + t] = acc[j][k];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Windowed form (the default where its windows fit): a CTA owns D DM trials x
// kDdThreads * P output samples.  Per channel, the window of input samples
// its trials read -- from the tile's smallest to its largest delay -- is
// brought into shared memory by one bulk asynchronous copy, kDwC channels a
// stage in a ring of kDwS stages (full: an mbarrier per stage; empty: one CTA
// barrier per stage), and every copied sample serves all D trials.  The sums
// are the same rounded float adds in the same channel order as k_dedisperse.
//
// A bulk copy starts on a 16-byte boundary: the host rounds each window's
// start down and adds the remainder (0..3 samples, the same for every time
// tile) to the trials' offsets.  A window whose rounded range would leave
// the filterbank (the last channel's end, a first row at an odd address) is
// copied sample by sample instead.
//
// Every addition reads its sample from shared memory, so the kernel is bound
// by the shared-memory pipe: at one 128-byte wavefront per clock 3.4e10
// additions (1024 channels, 128 trials, 2^18 samples) take 3.4 ms.  With the
// windows copied by 4-byte cp.async and 32-bit offsets read one at a time,
// those took a fifth of the pipe and a CTA-wide wait every 8 channels: 6.1 ms;
// this form 4.4 ms (77 % of that bound).  Two stages of 8 channels measured the
// same here and 1.63 against 1.34 ms at 300 channels and a DM step of 3; three
// CTAs per SM (85 registers) 4.7 ms.
constexpr int kDwC = 4;   // channels per stage
constexpr int kDwS = 3;   // stages
constexpr size_t kDwSmemMax = 110 * 1024;  // two CTAs per SM

constexpr int kDwT = kDdThreads * kDdPer;  // output samples per CTA

__device__ __forceinline__ float2 add2_rn(float2 a, float2 b) {
    float2 r;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 x, x, y;\n"
        " mov.b64 {%0, %1}, x;\n}\n"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// The tile's outputs of one thread, each sample read from global memory:
// start and offs are the tile's, t the thread's first output sample.
template <int D>
__device__ __noinline__ void dw_tile_from_global(const float* __restrict__ in, int nchan,
                                                 const long long* __restrict__ start,
                                                 const unsigned short* __restrict__ offs, long long t, int nd,
                                                 float* __restrict__ out, long long nout) {
#pragma unroll 1
    for (int j = 0; j < nd; j++)
#pragma unroll 1
        for (int q = 0; q < kDdPer; q++) {
            const long long tq = t + (long long)q * kDdThreads;
            if (tq >= nout) break;
            float s = 0.f;
#pragma unroll 1
            for (int c = 0; c < nchan; c++) s = __fadd_rn(s, __ldg(in + start[c] + offs[c * D + j] / 4 + tq));
            out[(long long)j * nout + tq] = s;
        }
}

template <int D>
__global__ void __launch_bounds__(kDdThreads, 2)
    k_dedisperse_win(const float* __restrict__ in, int nchan, long long total, const long long* __restrict__ start,
                     const unsigned short* __restrict__ offs, int ndm, int ndtile, int wlen, float* __restrict__ out,
                     long long nout, unsigned test_extra_tx) {
    constexpr int P = kDdPer;
    extern __shared__ __align__(128) float dsm[];  // [kDwS][kDwC][wlen] windows, then [kDwS][kDwC][D] offsets
    unsigned short* soff = reinterpret_cast<unsigned short*>(dsm + kDwS * kDwC * wlen);
    __shared__ __align__(8) unsigned long long full[kDwS];
    const long long bid = blockIdx.x;
    const int tile = (int)(bid % ndtile);
    const int d0 = tile * D;
    const long long t0 = (bid / ndtile) * (long long)kDwT;
    const int tid = threadIdx.x;
    const int nstage = (nchan + kDwC - 1) / kDwC;
    if (tid == 0)
        for (int s = 0; s < kDwS; s++) mbar_init(&full[s], 1);
    __syncthreads();
    // fill the ring slot of stage k (every thread calls it)
    auto fill = [&](int k) {
        const int slot = k % kDwS, c0 = k * kDwC, nc = min(kDwC, nchan - c0);
        const long long* __restrict__ st = start + (long long)tile * nchan + c0;
        unsigned bytes = 0;
        for (int cc = 0; cc < nc; cc++) {
            const long long at = st[cc] + t0;
            if (at >= 0 && at + wlen <= total) {
                bytes += 4u * (unsigned)wlen;
            } else {  // uniform: this window leaves the filterbank
                float* dst = dsm + (slot * kDwC + cc) * wlen;
                for (int x = tid; x < wlen; x += kDdThreads)
                    dst[x] = at + x >= 0 && at + x < total ? in[at + x] : 0.f;
            }
        }
        if (tid == 0) {
            // samples copied one by one for this slot's earlier stages come
            // before the bulk writes
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            constexpr unsigned ob = 2u * D * kDwC;
            mbar_arrive_expect_tx(&full[slot], bytes + ob + test_extra_tx);
            bulk_copy_g2s(soff + slot * kDwC * D, offs + ((long long)tile * nstage + k) * kDwC * D, ob, &full[slot]);
            for (int cc = 0; cc < nc; cc++) {
                const long long at = st[cc] + t0;
                if (at >= 0 && at + wlen <= total)
                    bulk_copy_g2s(dsm + (slot * kDwC + cc) * wlen, in + at, 4u * (unsigned)wlen, &full[slot]);
            }
        }
    };
    float2 acc[D][P / 2];
#pragma unroll
    for (int j = 0; j < D; j++)
#pragma unroll
        for (int q = 0; q < P / 2; q++) acc[j][q] = make_float2(0.f, 0.f);
    for (int k = 0; k < kDwS - 1 && k < nstage; k++) fill(k);
    int landed = 1;
    int k = 0;
#pragma unroll 1
    for (; k < nstage; k++) {
        const int slot = k % kDwS;
        // everyone is done with stage k - 1 (its slot is refilled now), sees
        // the samples copied one by one for stage k, and agrees on whether
        // stage k - 1 had landed: either all go on or all leave here
        if (!__syncthreads_and(landed)) break;
        if (k + kDwS - 1 < nstage) fill(k + kDwS - 1);
        landed = mbar_wait_bounded(&full[slot], (unsigned)(k / kDwS) & 1u);
        if (!landed) continue;
        const int nc = min(kDwC, nchan - k * kDwC);
#pragma unroll 2
        for (int cc = 0; cc < nc; cc++) {
            const char* w = reinterpret_cast<const char*>(dsm + (slot * kDwC + cc) * wlen + tid);
            const uint2* op = reinterpret_cast<const uint2*>(soff + (slot * kDwC + cc) * D);
#pragma unroll
            for (int j4 = 0; j4 < D / 4; j4++) {
                const uint2 o = op[j4];
                const unsigned off[4] = {o.x & 0xffffu, o.x >> 16, o.y & 0xffffu, o.y >> 16};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float* v = reinterpret_cast<const float*>(w + off[j]);
#pragma unroll
                    for (int q = 0; q < P / 2; q++)
                        acc[4 * j4 + j][q] = add2_rn(acc[4 * j4 + j][q],
                                                     make_float2(v[2 * q * kDdThreads], v[(2 * q + 1) * kDdThreads]));
                }
            }
        }
    }
    if (!__syncthreads_and(landed)) {
        // A copy did not land within the wait's limit (stage k - 1; up to
        // kDwS - 1 later ones are in flight: a last chance for all of them).
        // The call has returned long ago and has no status left to give, so
        // the tile is summed from global memory instead: the same samples in
        // the same order.
        for (int m = k - 1; m < nstage && m < k - 1 + kDwS; m++)
            mbar_wait_bounded(&full[m % kDwS], (unsigned)(m / kDwS) & 1u);
        dw_tile_from_global<D>(in, nchan, start + (long long)tile * nchan, offs + (long long)tile * nstage * kDwC * D,
                               t0 + tid, min(D, ndm - d0), out + (long long)d0 * nout, nout);
        return;
    }
#pragma unroll
    for (int j = 0; j < D; j++) {
        if (d0 + j < ndm) {
#pragma unroll
            for (int q = 0; q < P; q++) {
                const long long t = t0 + tid + (long long)q * kDdThreads;
                if (t < nout) out[(long long)(d0 + j) * nout + t] = (q & 1) ? acc[j][q / 2].y : acc[j][q / 2].x;
            }
        }
    }
}

// Tables of the windowed form: window starts [ndtile][nchan], then (16-byte
// aligned) the trials' byte offsets [ndtile][whole stages of channels][D].
// Filling them is the call's host work, and with many trials of short outputs
// most of its time: every loop below runs along the channels.  (1024 channels x
// 2048 trials x 4096 samples 3.8 ms; with a pass over the delays for each tile
// height and the offsets filled down the trials 8.9; with 32-bit delays relative
// to 16-trial tiles, as the windows were copied sample by sample, 5.7.)
struct DwPlan {
    int ndtile = 0, wlen = 0;
    size_t offs_at = 0, bytes = 0;
    std::unique_ptr<char[]> tab;
};

static size_t dw_smem(int D, int wlen) { return sizeof(float) * kDwS * kDwC * (size_t)wlen + 2 * kDwS * kDwC * D; }

// Smallest and largest delay of every channel over tiles of 4, 8 and 16 trials.
struct DwBounds {
    std::vector<int> lo[3], hi[3];  // [tile][nchan]
    int spread[3];                  // widest range of a channel within a tile
};

static void dw_bounds(DwBounds& b, const int* delays, int nchan, int ndm) {
    for (int k = 0; k < 3; k++) {
        const int D = 4 << k, nt = (ndm + D - 1) / D, parts = k ? (ndm + D / 2 - 1) / (D / 2) : ndm, per = k ? 2 : 4;
        const int* lo_in = k ? b.lo[k - 1].data() : delays;
        const int* hi_in = k ? b.hi[k - 1].data() : delays;
        b.lo[k].resize((size_t)nt * nchan);
        b.hi[k].resize((size_t)nt * nchan);
        int spread = 0;
        for (int t = 0; t < nt; t++) {
            int* lo = b.lo[k].data() + (size_t)t * nchan;
            int* hi = b.hi[k].data() + (size_t)t * nchan;
            std::copy(lo_in + (size_t)t * per * nchan, lo_in + ((size_t)t * per + 1) * nchan, lo);
            std::copy(hi_in + (size_t)t * per * nchan, hi_in + ((size_t)t * per + 1) * nchan, hi);
            for (int j = t * per + 1; j < std::min(parts, (t + 1) * per); j++) {
                const int* l = lo_in + (size_t)j * nchan;
                const int* h = hi_in + (size_t)j * nchan;
                for (int c = 0; c < nchan; c++) {
                    lo[c] = std::min(lo[c], l[c]);
                    hi[c] = std::max(hi[c], h[c]);
                }
            }
            for (int c = 0; c < nchan; c++) spread = std::max(spread, hi[c] - lo[c]);
        }
        b.spread[k] = spread;
    }
}

// k: the tile height is D = 4 << k.
static void dw_plan(DwPlan& p, const DwBounds& b, const float* in, const int* delays, int nchan, long long nsamp,
                    int ndm, int k, int wlen) {
    const int D = 4 << k, Q = D / 4;
    p.ndtile = (ndm + D - 1) / D;
    p.wlen = wlen;
    const size_t pad = (size_t)(nchan + kDwC - 1) / kDwC * kDwC;  // whole stages: 16-byte rows to copy
    p.offs_at = (sizeof(long long) * p.ndtile * nchan + 15) & ~(size_t)15;
    p.bytes = p.offs_at + sizeof(unsigned short) * p.ndtile * pad * D;
    p.tab.reset(new char[p.bytes]);
    const long long skew = (long long)((reinterpret_cast<uintptr_t>(in) >> 2) & 3);
    std::vector<int> base(nchan);             // sample offset of delay 0 in the window
    std::vector<unsigned long long> four(nchan);
    for (int tl = 0; tl < p.ndtile; tl++) {
        const int* lo = b.lo[k].data() + (size_t)tl * nchan;
        long long* start = reinterpret_cast<long long*>(p.tab.get()) + (size_t)tl * nchan;
        for (int c = 0; c < nchan; c++) {
            const long long at = (long long)c * nsamp + lo[c];
            const int rem = (int)((at + skew) & 3);
            start[c] = at - rem;
            base[c] = rem - lo[c];
        }
        // four trials' 16-bit offsets at a time as one 64-bit word (little-endian)
        char* row = p.tab.get() + p.offs_at + sizeof(unsigned short) * tl * pad * D;
        for (int q = 0; q < Q; q++) {
            const int d0 = tl * D + 4 * q;
            for (int j = 0; j < 4; j++) {
                if (d0 + j < ndm) {
                    const int* dl = delays + (size_t)(d0 + j) * nchan;
                    for (int c = 0; c < nchan; c++) {
                        const unsigned long long v = (unsigned)(4 * (dl[c] + base[c]));
                        four[c] = j ? four[c] | v << (16 * j) : v;
                    }
                } else if (j == 0) {
                    std::fill(four.begin(), four.end(), 0ull);  // padding trials
                }
            }
            for (int c = 0; c < nchan; c++) std::memcpy(row + 8 * ((size_t)c * Q + q), &four[c], 8);
        }
        std::memset(row + 8 * (size_t)nchan * Q, 0, 8 * (pad - nchan) * Q);
    }
}

template <int D>
static cudaError_t dw_launch(const DwPlan& p, const float* in, int nchan, long long nsamp, const char* tab, int ndm,
                             float* out, long long nout, bool wait_test, cudaStream_t st) {
    static std::atomic<unsigned long long> attr{0};
    int dev = 0;
    if (attr_pending(attr, &dev)) {
        cudaError_t e = cudaFuncSetAttribute(k_dedisperse_win<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kDwSmemMax);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_dedisperse_win<D>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        attr_set(attr, dev);
    }
    const long long ntt = (nout + kDwT - 1) / kDwT;
    k_dedisperse_win<D><<<(unsigned)(p.ndtile * ntt), kDdThreads, dw_smem(D, p.wlen), st>>>(
        in, nchan, (long long)nchan * nsamp, reinterpret_cast<const long long*>(tab),
        reinterpret_cast<const unsigned short*>(tab + p.offs_at), ndm, p.ndtile, p.wlen, out, nout,
        wait_test ? 16u : 0u);
    return cudaGetLastError();
}

}  // namespace accel

using namespace accel;

static int dedisperse(const float* filterbank_dev, int nchan, long long nsamp, const int* delays, int ndm,
                      float* out_dev, long long nout, bool wait_test, void* cuda_stream) {
    if (!filterbank_dev || !out_dev || !delays || nchan < 1 || ndm < 1 || nsamp < 1 || nout < 1)
        return set_error(ACCEL_ERR_INVALID, "accel_dedisperse: bad argument");
    const long long nd = (long long)ndm * nchan;
    int mn = 0, mx = 0;
    for (long long i = 0; i < nd; i++) {
        mn = std::min(mn, delays[i]);
        mx = std::max(mx, delays[i]);
    }
    if (mn < 0) return set_error(ACCEL_ERR_INVALID, "accel_dedisperse: negative delay");
    if (nout > nsamp - mx)
        return set_error(ACCEL_ERR_INVALID, "accel_dedisperse: %lld output samples need %lld input samples, have %lld",
                         nout, nout + mx, nsamp);
    cudaStream_t st = (cudaStream_t)cuda_stream;
    const long long ntt = (nout + kDdThreads * kDdPer - 1) / (kDdThreads * kDdPer);
    {
        // windowed kernel: the tile height that pads and copies least among
        // those whose windows fit
        DwBounds bounds;
        dw_bounds(bounds, delays, nchan, ndm);
        int D = 0, wlen = 0, height = 0;
        double best = 0;
        for (int k : {2, 1, 0}) {
            const int d = 4 << k;
            const long long spread = bounds.spread[k], need = (kDwT + spread + 3 + 3) & ~3LL;
            const long long nt = (ndm + d - 1) / d;
            if (4 * (spread + 3) > 65535 || dw_smem(d, (int)need) > kDwSmemMax || nt * ntt > 0x7fffffffLL) continue;
            const double cost = (double)nt * d * (1.0 + (double)need / ((double)kDwT * d));
            if (!D || cost < best) D = d, height = k, wlen = (int)need, best = cost;
        }
        if (D) {
            DwPlan p;
            dw_plan(p, bounds, filterbank_dev, delays, nchan, nsamp, ndm, height, wlen);
            char* d_tab = nullptr;
            cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&d_tab), p.bytes, st);
            // from pageable memory: staged before the call returns
            if (e == cudaSuccess) e = cudaMemcpyAsync(d_tab, p.tab.get(), p.bytes, cudaMemcpyHostToDevice, st);
            if (e == cudaSuccess)
                e = D == 16  ? dw_launch<16>(p, filterbank_dev, nchan, nsamp, d_tab, ndm, out_dev, nout, wait_test, st)
                    : D == 8 ? dw_launch<8>(p, filterbank_dev, nchan, nsamp, d_tab, ndm, out_dev, nout, wait_test, st)
                             : dw_launch<4>(p, filterbank_dev, nchan, nsamp, d_tab, ndm, out_dev, nout, wait_test, st);
            if (d_tab) {
                const cudaError_t ef = cudaFreeAsync(d_tab, st);
                if (e == cudaSuccess) e = ef;
            }
            if (e != cudaSuccess) return set_error(ACCEL_ERR_CUDA, "accel_dedisperse: %s", cudaGetErrorString(e));
            return ACCEL_OK;
        }
    }
    // delays too far apart within a tile for the windows: one load per addition
    const int ndtile = (ndm + kDdD - 1) / kDdD;
    if ((long long)ndtile * ntt > 0x7fffffffLL) return set_error(ACCEL_ERR_UNSUPPORTED, "accel_dedisperse: grid too large");
    // the kernel's table: channel-major, each channel's delays of all DM
    // trials padded to whole tiles of kDdD (one 32-byte sector per tile)
    const long long pad = (long long)ndtile * kDdD;
    std::vector<int> tab((size_t)(pad * nchan), 0);
    for (int d = 0; d < ndm; d++)
        for (int c = 0; c < nchan; c++) tab[(size_t)c * pad + d] = delays[(long long)d * nchan + c];
    int* d_delays = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&d_delays), sizeof(int) * tab.size(), st);
    if (e != cudaSuccess) return set_error(ACCEL_ERR_NOMEM, "accel_dedisperse: %s", cudaGetErrorString(e));
    // from pageable memory: staged before the call returns
    e = cudaMemcpyAsync(d_delays, tab.data(), sizeof(int) * tab.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        k_dedisperse<<<(unsigned)(ndtile * ntt), kDdThreads, 0, st>>>(
            filterbank_dev, nchan, nsamp, reinterpret_cast<const int4*>(d_delays), ndm, ndtile, out_dev, nout);
        e = cudaGetLastError();
    }
    const cudaError_t ef = cudaFreeAsync(d_delays, st);
    if (e == cudaSuccess) e = ef;
    if (e != cudaSuccess) return set_error(ACCEL_ERR_CUDA, "accel_dedisperse: %s", cudaGetErrorString(e));
    return ACCEL_OK;
}

extern "C" {

int accel_dedisperse_delays(int nchan, double f_top_mhz, double chan_bw_mhz, double tsamp, const float* dms,
                            int ndm, int* delays, int* max_delay) {
    if (nchan < 1 || ndm < 1 || !dms || !delays || !(tsamp > 0.0) || !(f_top_mhz > 0.0) || chan_bw_mhz == 0.0)
        return set_error(ACCEL_ERR_INVALID, "accel_dedisperse_delays: bad argument");
    const double f_last = f_top_mhz + (nchan - 1) * chan_bw_mhz;
    if (!(f_last > 0.0)) return set_error(ACCEL_ERR_INVALID, "accel_dedisperse_delays: channel frequency <= 0");
    const double f_ref = std::max(f_top_mhz, f_last);
    const double inv_ref2 = 1.0 / (f_ref * f_ref);
    int mx = 0;
    for (int d = 0; d < ndm; d++) {
        if (!(dms[d] >= 0.0f)) return set_error(ACCEL_ERR_INVALID, "accel_dedisperse_delays: DM %d < 0", d);
        for (int c = 0; c < nchan; c++) {
            const double f = f_top_mhz + c * chan_bw_mhz;
            const double v = std::floor(kDispConst * (double)dms[d] * (1.0 / (f * f) - inv_ref2) / tsamp + 0.5);
            if (v > 2147483647.0) return set_error(ACCEL_ERR_INVALID, "accel_dedisperse_delays: delay overflow");
            delays[(long long)d * nchan + c] = (int)v;
            mx = std::max(mx, (int)v);
        }
    }
    if (max_delay) *max_delay = mx;
    return ACCEL_OK;
}

int accel_dedisperse(const float* filterbank_dev, int nchan, long long nsamp, const int* delays, int ndm,
                     float* out_dev, long long nout, void* cuda_stream) {
    return dedisperse(filterbank_dev, nchan, nsamp, delays, ndm, out_dev, nout, false, cuda_stream);
}

int accel_dedisperse_wait_test(const float* filterbank_dev, int nchan, long long nsamp, const int* delays, int ndm,
                               float* out_dev, long long nout, void* cuda_stream) {
    return dedisperse(filterbank_dev, nchan, nsamp, delays, ndm, out_dev, nout, true, cuda_stream);
}

}  // extern "C"
