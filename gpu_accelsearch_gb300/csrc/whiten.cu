// whiten.cu -- red-noise removal (deredden, bpd_noise.c:12-92) on the GPU.
//
// The reference walks the spectrum serially: block medians of growing
// width (initialbuflen*ln(binnum), capped at maxbuflen), a linear slope
// between neighbouring block levels, and amplitude *= rsqrt(level).  The
// block boundaries are a serial recurrence and are planned on the host
// (plan_whiten_blocks in api.cu); everything else is parallel:
//   k_whiten_medians  one CTA per block: exact lower median of |A|^2
//                     (radix select), level = median / ln 2 in double;
//   k_whiten_scale    one CTA per write range: the range's level and slope
//                     from its two neighbouring blocks, then the scaling
//                     with the reference's float arithmetic.
// Results are bit-identical to the reference's host routine.
#include <cmath>
#include <mutex>

#include "../../include/accelsearch.h"
#include "accel_internal.h"

namespace accel {

constexpr double kLn2w = 0.693147180559945309417232121458;

__global__ void __launch_bounds__(256) k_whiten_medians(const int* __restrict__ bstart,
                                                        const int* __restrict__ blen,
                                                        const float2* __restrict__ spec, double* med) {
    extern __shared__ uint32_t keys[];
    __shared__ int hist[256];
    __shared__ int bc[2];
    const int b = blockIdx.x;
    const int s = bstart[b], n = blen[b];
    for (int i = threadIdx.x; i < n; i += blockDim.x) keys[i] = __float_as_uint(power_exact(spec[s + i]));
    __syncthreads();
    const uint32_t k = block_select_u32(keys, n, (n - 1) / 2, hist, bc);
    if (threadIdx.x == 0) med[b] = (double)__uint_as_float(k) / kLn2w;
}

// Write range r (0 <= r <= nb): r = 0 is the first half-block with a flat
// level; 1 <= r < nb interpolate from block r-1 towards block r; r = nb is
// the tail, continuing the last slope (1.0 when there was no second block).
__global__ void __launch_bounds__(256) k_whiten_scale(const int* __restrict__ bstart,
                                                      const int* __restrict__ blen,
                                                      const double* __restrict__ med, int nb,
                                                      float2* spec, unsigned numbins, int exact) {
    const int r = blockIdx.x;
    long long lo, hi;
    float mean_old, dslope;
    if (r == 0) {
        lo = 1;
        hi = bstart[0] + blen[0] / 2;
        mean_old = (float)med[0];
        dslope = 0.f;
        if (threadIdx.x == 0) spec[0] = make_float2(1.0f, 0.0f);
    } else if (r < nb) {
        lo = bstart[r - 1] + blen[r - 1] / 2;
        hi = bstart[r] + blen[r] / 2;
        mean_old = (float)med[r - 1];
        dslope = (float)((med[r] - (double)mean_old) / (0.5 * (blen[r - 1] + blen[r])));
    } else {
        lo = bstart[nb - 1] + blen[nb - 1] / 2;
        hi = numbins;
        mean_old = (float)med[nb - 1];
        if (nb >= 2) {
            const float mo = (float)med[nb - 2];
            dslope = (float)((med[nb - 1] - (double)mo) / (0.5 * (blen[nb - 2] + blen[nb - 1])));
        } else {
            dslope = 1.0f;
        }
    }
    const float flat = rsqrt_norm(mean_old, exact);
    for (long long ind = lo + threadIdx.x; ind < hi; ind += blockDim.x) {
        float norm;
        if (r == 0) norm = flat;
        else norm = rsqrt_norm(__fadd_rn(mean_old, __fmul_rn(dslope, (float)(ind - lo))), exact);
        float2 v = spec[ind];
        v.x = __fmul_rn(v.x, norm);
        v.y = __fmul_rn(v.y, norm);
        spec[ind] = v;
    }
}

// Forms of the two kernels for blocks of at most kWarpBlockMax bins (the
// reference's widths are at most 200): a warp per block or range, eight
// warps per CTA, no keys or histograms in shared memory.
//
// Both are one pass over the spectrum (8 and 16 bytes per bin) and should be
// bound by memory.  The first form was not: a digit histogram per warp in
// shared memory (match_any and atomics for every key), and one
// double-precision division per warp -- all 32 lanes of it, at 1/64 of the
// single-precision rate -- for every level and slope.  Now the median is a
// bitwise search over keys in registers (counts by redux.sync, stopped when
// one key is left in the interval) and levels and slopes are computed by one
// lane per range.  2^21 bins, GB300: medians 55 -> 12 us, scaling 31 -> 11 us
// (cold cache).
constexpr int kWarpBlockMax = 1024;
constexpr int kWarpsPerCta = 8;
constexpr int kScaleRanges = 32;  // write ranges per CTA of the scaling kernel
constexpr int kScaleWarps = 16;

// Lower median (rank (n - 1) / 2, 0-based) of the warp's n keys, lane l
// holding keys l, l + 32, ... in key[], unused slots 0xffffffff.
template <int NK>
__device__ __forceinline__ uint32_t warp_median(const uint32_t (&key)[NK], int n) {
    const int lane = threadIdx.x & 31;
    uint32_t any = 0, all = 0xffffffffu;  // bits set in some key, in every key
#pragma unroll
    for (int j = 0; j < NK; j++)
        if (lane + 32 * j < n) {
            any |= key[j];
            all &= key[j];
        }
    any = __reduce_or_sync(0xffffffffu, any);
    all = __reduce_and_sync(0xffffffffu, all);
    const uint32_t diff = any ^ all;
    if (diff == 0) return all;  // all keys equal
    const int k = (n - 1) / 2;
    int bit = 31 - __clz(diff);
    uint32_t lo = bit == 31 ? 0u : all & ~((2u << bit) - 1u);  // the keys' common leading bits
    int below = 0, upto = n;  // keys < lo, keys < lo + 2^(bit + 1)
#pragma unroll 1
    for (; bit >= 0 && upto - below > 1; bit--) {
        const uint32_t mid = lo | (1u << bit);
        int c = 0;
#pragma unroll
        for (int j = 0; j < NK; j++) c += key[j] < mid;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c <= k) {
            lo = mid;
            below = c;
        } else {
            upto = c;
        }
    }
    if (bit < 0) return lo;
    // one key left in [lo, lo + 2^(bit + 1))
    const uint32_t lead = lo >> bit >> 1;
    uint32_t mine = 0;
#pragma unroll
    for (int j = 0; j < NK; j++)
        if (lane + 32 * j < n && (key[j] >> bit >> 1) == lead) mine = key[j];
    return __reduce_or_sync(0xffffffffu, mine);
}

// med[b]: the block's median power (the level's division is left to the
// scaling kernel).  NK: registers for the widest block, 32 NK bins; with the
// widths of one call known, a warp carries no more registers than it needs
// (32 keys in every warp held the kernel at 32 warps per SM).
template <int NK>
__global__ void __launch_bounds__(32 * kWarpsPerCta) k_whiten_medians_warp(const int* __restrict__ bstart,
                                                                           const int* __restrict__ blen,
                                                                           const float2* __restrict__ spec,
                                                                           float* __restrict__ med, int nblocks) {
    const int b = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (b >= nblocks) return;
    const int lane = threadIdx.x & 31, n = blen[b];
    const float2* __restrict__ s = spec + bstart[b];
    uint32_t key[NK];
#pragma unroll
    for (int j = 0; j < NK; j++) {
        const int i = lane + 32 * j;
        key[j] = i < n ? __float_as_uint(power_exact(s[i])) : 0xffffffffu;
    }
    const uint32_t k = warp_median<NK>(key, n);
    if (lane == 0) med[b] = __uint_as_float(k);
}

template <int NK>
static void launch_medians(const int* bstart, const int* blen, const float2* spec, float* med, int nblocks,
                           cudaStream_t st) {
    k_whiten_medians_warp<NK><<<(nblocks + kWarpsPerCta - 1) / kWarpsPerCta, 32 * kWarpsPerCta, 0, st>>>(
        bstart, blen, spec, med, nblocks);
}

// Write ranges as in k_whiten_scale, kScaleRanges per CTA: their starts,
// levels and slopes by one thread each, then a warp per range.
__global__ void __launch_bounds__(32 * kScaleWarps) k_whiten_scale_warp(const int* __restrict__ bstart,
                                                                         const int* __restrict__ blen,
                                                                         const float* __restrict__ med, int nb,
                                                                         float2* spec, unsigned numbins,
                                                                         int exact) {
    __shared__ int s_lo[kScaleRanges + 1];
    __shared__ float s_mean[kScaleRanges], s_slope[kScaleRanges];
    __shared__ double s_level[kScaleRanges + 1];
    const int r0 = blockIdx.x * kScaleRanges, nr = min(kScaleRanges, nb + 1 - r0);
    // levels of blocks first .. first + nr (the tail also looks one block back)
    const int first = max(0, min(r0 - 1, nb - 2)), i = threadIdx.x;
    if (i <= kScaleRanges && first + i < nb) s_level[i] = (double)med[first + i] / kLn2w;
    if (i <= nr) {
        const int r = r0 + i;
        s_lo[i] = r == 0 ? 1 : r <= nb ? bstart[r - 1] + blen[r - 1] / 2 : (int)numbins;
    }
    __syncthreads();
    if (i < nr) {
        const int r = r0 + i;
        auto level = [&](int b) { return s_level[b - first]; };
        float mean_old, dslope = 0.f;
        if (r == 0) {
            mean_old = (float)level(0);
            spec[0] = make_float2(1.0f, 0.0f);
        } else if (r < nb) {
            mean_old = (float)level(r - 1);
            dslope = (float)((level(r) - (double)mean_old) / (0.5 * (blen[r - 1] + blen[r])));
        } else {
            mean_old = (float)level(nb - 1);
            if (nb >= 2) {
                const float mo = (float)level(nb - 2);
                dslope = (float)((level(nb - 1) - (double)mo) / (0.5 * (blen[nb - 2] + blen[nb - 1])));
            } else {
                dslope = 1.0f;
            }
        }
        s_mean[i] = mean_old;
        s_slope[i] = dslope;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int q = threadIdx.x >> 5; q < nr; q += kScaleWarps) {
        const unsigned lo = (unsigned)s_lo[q], hi = (unsigned)s_lo[q + 1];
        const float mean_old = s_mean[q], dslope = s_slope[q];
        if (r0 + q == 0) {
            const float flat = rsqrt_norm(mean_old, exact);
            for (unsigned ind = lo + lane; ind < hi; ind += 32) {
                const float2 v = spec[ind];
                spec[ind] = make_float2(__fmul_rn(v.x, flat), __fmul_rn(v.y, flat));
            }
            continue;
        }
        // four bins per lane in flight
#pragma unroll 1
        for (unsigned at = lo + lane; at < hi; at += 128) {
            float2 v[4];
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (at + 32 * j < hi) v[j] = spec[at + 32 * j];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const unsigned ind = at + 32 * j;
                if (ind >= hi) break;
                const float norm = rsqrt_norm(__fadd_rn(mean_old, __fmul_rn(dslope, (float)(ind - lo))), exact);
                spec[ind] = make_float2(__fmul_rn(v[j].x, norm), __fmul_rn(v[j].y, norm));
            }
        }
    }
}

// Block recurrence of deredden (bpd_noise.c:33-79): the first block holds
// initbuf bins from bin 1; each next block starts where the last ended and
// holds (int)(initbuf * ln(start)) bins, at most maxbuf; blocks continue
// while start + length < numbins.  Positions are carried in 64 bits so that
// no sum overflows near kMaxWhitenBins; the width is clamped before the
// conversion to int (same result wherever the reference's is defined).
long long whiten_blocks(long long numbins, int initbuf, int maxbuf, int* start, int* len, long long cap) {
    if (initbuf < 1 || maxbuf < 1 || numbins <= 1 + (long long)initbuf || numbins > kMaxWhitenBins) return -1;
    auto width = [&](long long at) {
        const double x = initbuf * std::log((double)at);
        return x >= (double)maxbuf ? maxbuf : (int)x;
    };
    long long n = 0, binnum = 1;
    int buflen = initbuf;
    for (;;) {
        if (n < cap) {
            start[n] = (int)binnum;
            len[n] = buflen;
        }
        n++;
        binnum += buflen;
        buflen = width(binnum);
        if (binnum + buflen >= numbins) break;
    }
    return n;
}

std::vector<std::pair<int, int>> plan_whiten_blocks(long long numbins, int initbuf, int maxbuf) {
    const long long n = whiten_blocks(numbins, initbuf, maxbuf, nullptr, nullptr, 0);
    std::vector<std::pair<int, int>> b;
    if (n <= 0) return b;
    std::vector<int> s((size_t)n), l((size_t)n);
    whiten_blocks(numbins, initbuf, maxbuf, s.data(), l.data(), n);
    b.reserve((size_t)n);
    for (long long i = 0; i < n; i++) b.push_back({s[i], l[i]});
    return b;
}

int launch_whiten(const int* d_bstart, const int* d_blen, int nblocks, double* d_med, float2* spec,
                  unsigned numbins, int maxlen, cudaStream_t st, int exact) {
    if (maxlen <= kWarpBlockMax) {
        float* med = reinterpret_cast<float*>(d_med);
        // widths at the default cap: 78 at 2^18 bins, 87 at 2^21, 99 at 2^24
        if (maxlen <= 64) launch_medians<2>(d_bstart, d_blen, spec, med, nblocks, st);
        else if (maxlen <= 96) launch_medians<3>(d_bstart, d_blen, spec, med, nblocks, st);
        else if (maxlen <= 128) launch_medians<4>(d_bstart, d_blen, spec, med, nblocks, st);
        else if (maxlen <= 256) launch_medians<8>(d_bstart, d_blen, spec, med, nblocks, st);
        else launch_medians<kWarpBlockMax / 32>(d_bstart, d_blen, spec, med, nblocks, st);
        if (cudaGetLastError() != cudaSuccess) return -1;
        k_whiten_scale_warp<<<nblocks / kScaleRanges + 1, 32 * kScaleWarps, 0, st>>>(d_bstart, d_blen, med, nblocks, spec,
                                                                                   numbins, exact);
        return cudaGetLastError() == cudaSuccess ? 0 : -1;
    }
    size_t smem = sizeof(uint32_t) * (size_t)maxlen;
    if (smem > 48 * 1024) {
        if (cudaFuncSetAttribute(k_whiten_medians, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess)
            return -1;
    }
    k_whiten_medians<<<nblocks, 256, smem, st>>>(d_bstart, d_blen, spec, d_med);
    if (cudaGetLastError() != cudaSuccess) return -1;
    k_whiten_scale<<<nblocks + 1, 256, 0, st>>>(d_bstart, d_blen, d_med, nblocks, spec, numbins, exact);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace accel

// --------------------------------------------------------------------------
// Allocation-free whitening (accel_whiten_noalloc).
//
// Same kernels as above; their scratch -- the block table (start, length)
// and the per-block levels -- lives in one file-scope device array instead
// of memory allocated by a context.  Every GPU that loads the library holds
// this array (2 MiB) until the process exits.  All calls share it, so calls
// whose GPU work overlaps race; every byte a call reads is written earlier
// by the same call (table copy, then medians), so nothing needs clearing.
namespace accel {
namespace {

constexpr int kNoAllocBlocks = 131072;
constexpr size_t kNoAllocBytes = (size_t)kNoAllocBlocks * (2 * sizeof(int) + sizeof(double));
static __device__ __align__(256) unsigned char g_whiten_scratch[kNoAllocBytes];

constexpr int kNoAllocDevices = 64;
std::mutex g_noalloc_mutex;
void* g_noalloc_addr[kNoAllocDevices];           // device address of g_whiten_scratch
int g_noalloc_start[kNoAllocBlocks];             // host staging of the block table
int g_noalloc_len[kNoAllocBlocks];

}  // namespace
}  // namespace accel

extern "C" int accel_whiten_noalloc(accel_complex* spec, long long numbins, int initbuf, int maxbuf,
                                    void* stream) {
    using namespace accel;
    if (!spec) return set_error(ACCEL_ERR_INVALID, "accel_whiten_noalloc: null spectrum");
    if (initbuf < 1 || maxbuf < 1 || maxbuf > 49152)
        return set_error(ACCEL_ERR_INVALID,
                         "accel_whiten_noalloc: block widths must be in [1, 49152]");
    if (numbins <= 1 + (long long)initbuf || numbins > kMaxWhitenBins)
        return set_error(ACCEL_ERR_INVALID, "accel_whiten_noalloc: %lld bins out of range (%d .. %lld)",
                         numbins, initbuf + 2, kMaxWhitenBins);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess)
        return set_error(ACCEL_ERR_CUDA, "accel_whiten_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev < 0 || dev >= kNoAllocDevices)
        return set_error(ACCEL_ERR_UNSUPPORTED, "accel_whiten_noalloc: device %d", dev);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // The block table goes to the device by a copy from host arrays that the
    // next call overwrites: a captured copy would replay whatever table the
    // latest call left there, so calls inside a stream capture are refused.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    e = cudaStreamIsCapturing(st, &cap);
    if (e != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        if (e != cudaSuccess) cudaGetLastError();
        return set_error(ACCEL_ERR_UNSUPPORTED, "accel_whiten_noalloc: not callable during stream capture");
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_addr[dev]) {
        // once per device, with that device current: the array's device address
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_whiten_scratch);
        if (e != cudaSuccess || !p)
            return set_error(ACCEL_ERR_CUDA, "accel_whiten_noalloc: cudaGetSymbolAddress: %s",
                             cudaGetErrorString(e));
        g_noalloc_addr[dev] = p;
    }
    const long long nbl = whiten_blocks(numbins, initbuf, maxbuf, g_noalloc_start, g_noalloc_len, kNoAllocBlocks);
    const int nb = (int)nbl;
    if (nbl > kNoAllocBlocks)
        return set_error(ACCEL_ERR_INVALID,
                         "accel_whiten_noalloc: %lld bins need more than %d whitening blocks, the "
                         "size of the static scratch (about 1.2e7 bins with the default widths)",
                         numbins, kNoAllocBlocks);
    int maxlen = 0;
    for (int i = 0; i < nb; i++) maxlen = g_noalloc_len[i] > maxlen ? g_noalloc_len[i] : maxlen;
    char* base = static_cast<char*>(g_noalloc_addr[dev]);
    int* d_start = reinterpret_cast<int*>(base);
    int* d_len = reinterpret_cast<int*>(base + sizeof(int) * kNoAllocBlocks);
    double* d_med = reinterpret_cast<double*>(base + 2 * sizeof(int) * kNoAllocBlocks);
    // pageable source: the copies have left the host arrays when they return
    e = cudaMemcpyAsync(d_start, g_noalloc_start, sizeof(int) * nb, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(d_len, g_noalloc_len, sizeof(int) * nb, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess)
        return set_error(ACCEL_ERR_CUDA, "accel_whiten_noalloc: block table copy: %s",
                         cudaGetErrorString(e));
    if (launch_whiten(d_start, d_len, nb, d_med, reinterpret_cast<float2*>(spec), (unsigned)numbins,
                      maxlen, st) != 0)
        return set_error(ACCEL_ERR_CUDA, "accel_whiten_noalloc: launch: %s",
                         cudaGetErrorString(cudaGetLastError()));
    return ACCEL_OK;
}
