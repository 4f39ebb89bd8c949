// rfft.cu -- real-to-complex FFT of any even length N from power-of-two
// cuFFT plans only (the search's transform of a DM trial; the reference
// makes a cuFFT R2C plan of the trial's own length, bpd_fft.cu:4-48).
//
// The N real samples are read as K = N/2 complex values z[n] = x[2n] +
// i x[2n+1].  Z = DFT_K(z) is one power-of-two C2C transform when K is a
// power of two; when K = m L with L a power of two and an odd m <= 15, m
// transforms of L points (the samples j, j + m, j + 2m, ...) combined by
//     Z[k] = sum_j exp(-2 pi i j k / K) Y_j[k mod L]
// (one Cooley-Tukey step); else Bluestein's chirp-z form: with
// w[m] = exp(i pi m^2/K),
//     Z[k] = conj(w[k]) sum_n (z[n] conj(w[n])) w[k - n],
// a linear convolution done by power-of-two transforms of P >= 2K - 1
// points.  Every phase is a multiple of pi/K reduced exactly to r in
// [0, 2K) (m^2 mod 2K in integers) and evaluated as the double-precision
// product of two table entries, exp(i pi q S/K) exp(i pi t/K) with r = q S + t,
// S ~ sqrt(2K), rounded once to float.  The double-precision operations (1/64
// of the FP32 rate: the four per bin alone held the unpacking kernel at 15 us
// for K = 2^21, now 9) are done only where they can matter: the entries are
// kept as sums of two floats as well, multiplied with the products' rounding
// errors carried along, and only where that result lies so close to the middle
// of two floats that its own error could decide (3 in 100000) is the double
// product formed.  The N/2 + 1 bins follow from the transforms of the even and
// odd samples, E[k] = (Z[k] + conj Z[K-k]) / 2 and O[k] = (Z[k] - conj Z[K-k])
// / (2i):
//     X[k] = E[k] + exp(-2 pi i k / N) O[k],   k = 0 .. K   (Z[K] = Z[0]).
// A plan per power of two serves every length, so a stream of trials of
// many lengths (the serving path) makes no new cuFFT plan per trial --
// making one costs milliseconds of host time and holds up every other
// thread's CUDA calls while it runs.
//
// What depends on the length only -- the phase tables, Bluestein's chirp
// and the transform of its wrapped filter -- is laid out once per length and
// kept with the plans (the DM trials of an observation share one length),
// least recently used lengths leaving when more than kLengthBytes are held;
// the working arrays are kept too, and all of it goes back when an allocation
// of the context finds no memory (R2CEngine::release).  A call of Bluestein's form is then two
// power-of-two transforms instead of three, and at 2 x 609997 samples
// 74 us of kernels instead of 126 (cold cache).
#include <algorithm>
#include <iterator>
#include <map>

#include "context.h"

namespace accel {

namespace {

__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// Phase tables of exp(i pi r / K): entry t < S is exp(i pi t / K), entry
// S + q is exp(i pi q S / K) for q < ceil(2K/S); in double, and each component
// as a float (x, y) and what that rounding left (z, w).
__global__ void k_phase_tables(float4* __restrict__ tab, double2* __restrict__ dbl, long long K, int S, int nq) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S + nq) return;
    double s, c;
    if (i < S) sincospi((double)i / (double)K, &s, &c);
    else sincospi((double)(i - S) * (double)S / (double)K, &s, &c);
    const float ch = (float)c, sh = (float)s;
    tab[i] = make_float4(ch, sh, (float)(c - (double)ch), (float)(s - (double)sh));
    dbl[i] = make_double2(c, s);
}

struct Phase {
    const float4* tab;
    const double2* dbl;
    unsigned S, shift;  // S = 2^shift
    // exp(i pi r / K) for 0 <= r < 2K: the double product, rounded once
    __device__ __forceinline__ float2 operator()(unsigned r) const {
        bool sure;
        const float2 v = fast(r, sure);
        return sure ? v : exact(r);
    }
    // without double precision: the same value wherever sure is set
    __device__ __forceinline__ float2 fast(unsigned r, bool& sure) const {
        const float4 a = __ldg(tab + S + (r >> shift)), b = __ldg(tab + (r & (S - 1)));
        sure = true;
        return make_float2(diff_of_products(a.x, a.z, b.x, b.z, a.y, a.w, b.y, b.w, sure),
                           diff_of_products(a.x, a.z, b.y, b.w, -a.y, -a.w, b.x, b.z, sure));
    }
    __device__ __forceinline__ float2 exact(unsigned r) const {
        const double2 a = __ldg(dbl + S + (r >> shift)), b = __ldg(dbl + (r & (S - 1)));
        return make_float2((float)(a.x * b.x - a.y * b.y), (float)(a.x * b.y + a.y * b.x));
    }
    // the same with the plain float product (error about 1e-7)
    __device__ __forceinline__ float2 f(unsigned r) const {
        const float4 a = __ldg(tab + S + (r >> shift)), b = __ldg(tab + (r & (S - 1)));
        return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
    // (p + pl)(q + ql) - (u + ul)(v + vl) of two-float numbers.  The sum before
    // the last rounding is within 7 2^-48 of the exact value (entries 2^-48,
    // the neglected low product 2^-49, the additions 5.5 2^-48; 2^-45.9 is the
    // largest measured): where 2^-44 either way rounds alike, so does the
    // double product; elsewhere sure is cleared.
    static __device__ __forceinline__ float diff_of_products(float p, float pl, float q, float ql, float u, float ul,
                                                             float v, float vl, bool& sure) {
        const float m = __fmul_rn(p, q), n = __fmul_rn(u, v);
        const float me = __fmaf_rn(p, q, -m), ne = __fmaf_rn(u, v, -n);  // exact: m + me = p q
        const float d = __fsub_rn(m, n), t = __fsub_rn(d, m);
        const float de = __fsub_rn(__fsub_rn(m, __fsub_rn(d, t)), __fadd_rn(n, t));  // exact: d + de = m - n
        float low = __fadd_rn(de, __fsub_rn(me, ne));
        low = __fmaf_rn(p, ql, low);
        low = __fmaf_rn(pl, q, low);
        low = __fmaf_rn(-u, vl, low);
        low = __fmaf_rn(-ul, v, low);
        constexpr float kTol = 1.0f / (1ull << 44);
        sure = sure && __fadd_rn(d, __fadd_rn(low, kTol)) == __fadd_rn(d, __fsub_rn(low, kTol));
        return __fadd_rn(d, low);
    }
};

// T[j L + l] = z[j + m l]: the m subsequences of stride m, each contiguous
__global__ void k_ct_split(const float2* __restrict__ z, float2* __restrict__ T, int m, long long L) {
    const long long K = (long long)m * L;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < K;
         i += (long long)gridDim.x * blockDim.x) {
        const long long j = i / L, l = i - j * L;
        T[i] = z[j + (long long)m * l];
    }
}

// Z[k] = sum_j exp(-2 pi i j k / K) Y_j[k mod L], Y_j = T[j L .. j L + L)
__global__ void k_ct_combine(const float2* __restrict__ T, float2* __restrict__ Z, int m, long long L,
                             Phase ph) {
    const long long K = (long long)m * L;
    const unsigned long long K2 = 2ull * (unsigned long long)K;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < K;
         k += (long long)gridDim.x * blockDim.x) {
        const long long l = k & (L - 1);
        float2 acc = T[l];
        unsigned long long r = 0;  // 2 j k mod 2K, a multiple of pi/K
        for (int j = 1; j < m; j++) {
            r += 2ull * (unsigned long long)k;
            if (r >= K2) r -= K2;
            const float2 w = ph.f((unsigned)r);  // exp(+i pi r/K); the transform uses its conjugate
            const float2 y = T[(long long)j * L + l];
            acc.x += y.x * w.x + y.y * w.y;
            acc.y += y.y * w.x - y.x * w.y;
        }
        Z[k] = acc;
    }
}

// The chirp w[m] = exp(i pi m^2 / K), m in [0, K), wrapped to P points:
// b[m] and b[P - m], zero between.
__global__ void k_chirp(float2* __restrict__ b, long long K, long long P, Phase ph) {
    const unsigned long long K2 = 2ull * (unsigned long long)K;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P;
         i += (long long)gridDim.x * blockDim.x) {
        long long m = -1;
        if (i < K) m = i;
        else if (i > P - K) m = P - i;
        b[i] = m >= 0 ? ph((unsigned)(((unsigned long long)m * (unsigned long long)m) % K2)) : make_float2(0.f, 0.f);
    }
}

// a[n] = z[n] conj(w[n]) for n < K, zero up to P
__global__ void k_chirp_in(const float2* __restrict__ z, const float2* __restrict__ w, float2* __restrict__ a,
                           long long K, long long P) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = i < K ? cmulc(z[i], w[i]) : make_float2(0.f, 0.f);
}

__global__ void k_pointwise(float2* __restrict__ a, const float2* __restrict__ fb, long long P) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < P;
         i += (long long)gridDim.x * blockDim.x) {
        const float2 x = a[i], y = fb[i];
        a[i] = make_float2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
    }
}

// X[k] and X[K - k] from Z[k], Z[K - k] (k = 0: X[0] and X[K] from Z[0]).
__device__ __forceinline__ void unpack_pair(float2* __restrict__ X, long long K, long long k, float2 zk, float2 zc,
                                            const Phase& ph) {
    if (k == 0) {
        X[0] = make_float2(zk.x + zk.y, 0.f);
        X[K] = make_float2(zk.x - zk.y, 0.f);
        return;
    }
    // E = (Z[k] + conj Z[K-k]) / 2, O = (Z[k] - conj Z[K-k]) / (2i)
    const float2 e = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y - zc.y));
    const float2 o = make_float2(0.5f * (zk.y + zc.y), -0.5f * (zk.x - zc.x));
    auto put = [&](float2 v) {                    // v = exp(+i pi k / K) = exp(2 pi i k / N)
        const float2 t = make_float2(v.x, -v.y);  // exp(-2 pi i k / N)
        const float2 to = make_float2(t.x * o.x - t.y * o.y, t.x * o.y + t.y * o.x);
        X[k] = make_float2(e.x + to.x, e.y + to.y);
        // X[K-k] = conj(E) - conj(t) conj(O) = conj(E - t O)
        if (2 * k != K) X[K - k] = make_float2(e.x - to.x, -(e.y - to.y));
    };
    // (the rare other rounding stored afterwards: taken before, the branch
    // stood between the loop's loads: K = 2^21 took 6 us longer)
    bool sure;
    put(ph.fast((unsigned)k, sure));
    if (!sure) put(ph.exact((unsigned)k));
}

// In place over X[0 .. K]: Z[k] in X[k] on entry (k < K); thread k <= K/2
// writes X[k] and X[K - k].
__global__ void k_r2c_unpack(float2* __restrict__ X, long long K, Phase ph) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k <= K / 2;
         k += (long long)gridDim.x * blockDim.x)
        unpack_pair(X, K, k, X[k], X[k ? K - k : 0], ph);
}

// The same from Bluestein's convolution: Z[k] = conj(w[k]) y[k] / P (y: the
// unnormalised inverse transform, w: the chirp).
__global__ void k_chirp_unpack(const float2* __restrict__ y, const float2* __restrict__ w, float2* __restrict__ X,
                               long long K, float inv_p, Phase ph) {
    auto z = [&](long long i) {
        const float2 v = cmulc(y[i], w[i]);
        return make_float2(v.x * inv_p, v.y * inv_p);
    };
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k <= K / 2;
         k += (long long)gridDim.x * blockDim.x)
        unpack_pair(X, K, k, z(k), z(k ? K - k : 0), ph);
}

// Largest odd factor taken by the Cooley-Tukey step (its combine reads m
// values per output)
constexpr long long kCtMaxOdd = 15;

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    return (int)(g < 152 * 16 ? (g < 1 ? 1 : g) : 152 * 16);
}

}  // namespace

// What a length's transform keeps between calls.
struct R2CLength {
    void* mem = nullptr;        // phase tables, then (Bluestein) w and FB
    size_t bytes = 0;
    Phase ph{};
    float2* w = nullptr;        // chirp, K points
    float2* fb = nullptr;       // transform of the wrapped chirp, P points
    long long last_use = 0;
};

// Device memory kept for lengths, and for the working array; a call that
// needs more frees it again.
constexpr size_t kLengthBytes = (size_t)512 << 20;

R2CEngine::~R2CEngine() { clear(); }

void R2CEngine::clear() {
    for (auto& kv : plans) cufftDestroy(kv.second);
    plans.clear();
    for (auto& kv : lengths) {
        cudaFree(kv.second->mem);
        delete kv.second;
    }
    lengths.clear();
    length_bytes = 0;
    if (work) cudaFree(work);
    work = nullptr;
    work_bytes = 0;
}

// The forward/inverse C2C plan of P points (a power of two), made once.
static int c2c_plan(R2CEngine& e, long long P, cufftHandle* out) {
    auto it = e.plans.find(P);
    if (it != e.plans.end()) {
        *out = it->second;
        return 0;
    }
    cufftHandle h;
    if (cufftCreate(&h) != CUFFT_SUCCESS) return -1;
    long long n = P;
    size_t work = 0;
    if (cufftMakePlanMany64(h, 1, &n, nullptr, 1, P, nullptr, 1, P, CUFFT_C2C, 1, &work) != CUFFT_SUCCESS) {
        cufftDestroy(h);
        return -1;
    }
    e.plans[P] = h;
    *out = h;
    return 0;
}

// Bluestein's transform length of K points, 0 where K is a power of two or
// takes the Cooley-Tukey step.
static long long bluestein_points(long long K) {
    if ((K >> __builtin_ctzll(K)) <= kCtMaxOdd) return 0;
    long long P = 1;
    while (P < 2 * K - 1) P <<= 1;
    return P;
}

// Points of the transform's cuFFT plan, 0 where it uses none.
static long long plan_points(long long K) {
    if (const long long P = bluestein_points(K)) return P;
    const long long L = K & -K;
    return L > 1 || K == 1 ? L : 0;
}

static int exec_c2c(cufftHandle h, const float2* in, float2* out, int dir) {
    return cufftExecC2C(h, reinterpret_cast<cufftComplex*>(const_cast<float2*>(in)),
                        reinterpret_cast<cufftComplex*>(out), dir) == CUFFT_SUCCESS
               ? 0
               : -1;
}

// Lay out a length's tables on stream st (l.mem of l.bytes bytes allocated).
static int fill_length(R2CEngine& e, R2CLength& l, long long K, int S, int nq, int shift, cudaStream_t st) {
    float4* tab = static_cast<float4*>(l.mem);
    double2* dbl = reinterpret_cast<double2*>(tab + S + nq);
    l.ph = Phase{tab, dbl, (unsigned)S, (unsigned)shift};
    k_phase_tables<<<(S + nq + 255) / 256, 256, 0, st>>>(tab, dbl, K, S, nq);
    if (cudaGetLastError() != cudaSuccess) return -1;
    const long long P = bluestein_points(K);
    if (!P) return 0;
    l.w = reinterpret_cast<float2*>(dbl + S + nq);
    l.fb = l.w + K + (K & 1);
    cufftHandle h;
    if (c2c_plan(e, P, &h) || cufftSetStream(h, st) != CUFFT_SUCCESS) return -1;
    k_chirp<<<grid_for(P), 256, 0, st>>>(l.fb, K, P, l.ph);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(l.w, l.fb, sizeof(float2) * K, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return -1;
    return exec_c2c(h, l.fb, l.fb, CUFFT_FORWARD);
}

static void drop_length(R2CEngine& e, std::map<long long, R2CLength*>::iterator it, cudaStream_t st) {
    cudaFreeAsync(it->second->mem, st);
    e.length_bytes -= it->second->bytes;
    delete it->second;
    e.lengths.erase(it);
}

static void drop_work(R2CEngine& e, cudaStream_t st) {
    if (e.work) cudaFreeAsync(e.work, st);
    e.work = nullptr;
    e.work_bytes = 0;
}

// Everything kept but one length's tables, in stream order.
static void drop_others(R2CEngine& e, const R2CLength* in_use, cudaStream_t st) {
    for (auto it = e.lengths.begin(); it != e.lengths.end();) {
        auto next = std::next(it);
        if (it->second != in_use) drop_length(e, it, st);
        it = next;
    }
    drop_work(e, st);
}

void R2CEngine::release(cudaStream_t st) { drop_others(*this, nullptr, st); }

// Memory in stream order; when there is none, once more after giving back
// what is kept for other lengths and the working array (not in use while
// either is allocated).
static int alloc_on(R2CEngine& e, void** p, size_t bytes, cudaStream_t st, const R2CLength* in_use) {
    if (cudaMallocAsync(p, bytes, st) == cudaSuccess) return 0;
    cudaGetLastError();
    drop_others(e, in_use, st);
    if (cudaMallocAsync(p, bytes, st) == cudaSuccess) return 0;
    cudaGetLastError();
    *p = nullptr;
    return -2;
}

// The kept entry of half length K, made on first use.
static int length_entry(R2CEngine& e, long long K, cudaStream_t st, R2CLength** out) {
    auto it = e.lengths.find(K);
    if (it != e.lengths.end()) {
        it->second->last_use = ++e.clock;
        *out = it->second;
        return 0;
    }
    int shift = 0;
    while ((1LL << (2 * shift)) < 2 * K) shift++;
    const int S = 1 << shift, nq = (int)((2 * K + S - 1) / S);
    const long long P = bluestein_points(K);
    R2CLength* l = new R2CLength;
    l->bytes = (sizeof(float4) + sizeof(double2)) * (size_t)(S + nq) + (P ? sizeof(float2) * (size_t)(K + (K & 1) + P) : 0);
    // (a length too large to keep leaves again after the call)
    while (l->bytes <= kLengthBytes && e.length_bytes + l->bytes > kLengthBytes) {
        auto lru = e.lengths.begin();
        for (auto i = e.lengths.begin(); i != e.lengths.end(); ++i)
            if (i->second->last_use < lru->second->last_use) lru = i;
        drop_length(e, lru, st);
    }
    int rc = alloc_on(e, &l->mem, l->bytes, st, nullptr);
    if (rc) {
        delete l;
        return rc;
    }
    rc = fill_length(e, *l, K, S, nq, shift, st);
    if (rc) {
        cudaFreeAsync(l->mem, st);
        delete l;
        return rc;
    }
    l->last_use = ++e.clock;
    e.lengths[K] = l;
    e.length_bytes += l->bytes;
    *out = l;
    return 0;
}

// The transform with the length's tables l and working memory `work` (see
// work_points) on stream st.
static int r2c_with(R2CEngine& e, const R2CLength& l, const float2* z, long long K, float2* out, float2* work,
                    cudaStream_t st) {
    const int odd = (int)std::min<long long>(K >> __builtin_ctzll(K), kCtMaxOdd + 1);
    const long long P = bluestein_points(K);
    cufftHandle h = 0;
    if (P) {
        if (c2c_plan(e, P, &h) || cufftSetStream(h, st) != CUFFT_SUCCESS) return -1;
        k_chirp_in<<<grid_for(P), 256, 0, st>>>(z, l.w, work, K, P);
        if (cudaGetLastError() != cudaSuccess || exec_c2c(h, work, work, CUFFT_FORWARD)) return -1;
        k_pointwise<<<grid_for(P), 256, 0, st>>>(work, l.fb, P);
        if (cudaGetLastError() != cudaSuccess || exec_c2c(h, work, work, CUFFT_INVERSE)) return -1;
        k_chirp_unpack<<<grid_for(K / 2 + 1), 256, 0, st>>>(work, l.w, out, K, (float)(1.0 / (double)P), l.ph);
        return cudaGetLastError() == cudaSuccess ? 0 : -1;
    }
    const long long L = K / odd;
    if ((odd == 1 || L > 1) && (c2c_plan(e, L, &h) || cufftSetStream(h, st) != CUFFT_SUCCESS)) return -1;
    if (odd == 1) {
        if (exec_c2c(h, z, out, CUFFT_FORWARD)) return -1;
    } else {
        k_ct_split<<<grid_for(K), 256, 0, st>>>(z, work, odd, L);
        if (cudaGetLastError() != cudaSuccess) return -1;
        for (int j = 0; j < odd && L > 1; j++)
            if (exec_c2c(h, work + (long long)j * L, work + (long long)j * L, CUFFT_FORWARD)) return -1;
        k_ct_combine<<<grid_for(K), 256, 0, st>>>(work, out, odd, L, l.ph);
        if (cudaGetLastError() != cudaSuccess) return -1;
    }
    k_r2c_unpack<<<grid_for(K / 2 + 1), 256, 0, st>>>(out, K, l.ph);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Working memory of a transform: a row at an odd float offset is copied
// first (its samples are read as complex pairs); then Bluestein's or the
// Cooley-Tukey step's array.
static size_t work_points(long long K, bool misaligned) {
    const long long P = bluestein_points(K);
    const bool step = !P && (K & (K - 1));
    return (misaligned ? (size_t)K + (K & 1) : 0) + (size_t)(P ? P : step ? K : 0);
}

int r2c_any(R2CEngine& e, const float* x, long long n, float2* out, cudaStream_t st) {
    if (n < 2 || (n & 1)) return -1;
    const long long K = n / 2;
    const bool mis = (reinterpret_cast<uintptr_t>(x) & 7) != 0;
    const size_t wbytes = sizeof(float2) * work_points(K, mis);
    // Recorded into a caller's graph, the call keeps nothing: memory allocated
    // in a capture belongs to the graph, and a replay must not depend on
    // tables a later call may drop.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) {
        cudaGetLastError();
        cap = cudaStreamCaptureStatusNone;
    }
    const bool keep = cap == cudaStreamCaptureStatusNone;
    R2CEngine once;
    R2CEngine& owner = keep ? e : once;
    if (!keep) once.plans.swap(e.plans);  // plans are used either way
    // the plan first: when its work area finds no memory, once more after
    // giving back (and waiting: the plan's memory is not stream-ordered) what
    // is kept, of which nothing is in use yet
    R2CLength* l = nullptr;
    cufftHandle h;
    int rc = plan_points(K) ? c2c_plan(owner, plan_points(K), &h) : 0;
    if (rc && keep && e.held()) {
        cudaGetLastError();
        e.release(st);
        cudaStreamSynchronize(st);
        rc = c2c_plan(e, plan_points(K), &h);
    }
    if (!rc) rc = length_entry(owner, K, st, &l);
    void* work = nullptr;
    if (!rc && wbytes) {
        if (owner.work_bytes < wbytes) {
            drop_work(owner, st);
            rc = alloc_on(owner, &owner.work, wbytes, st, l);
            if (!rc) owner.work_bytes = wbytes;
        }
        work = owner.work;
    }
    if (!rc) {
        const float2* z = reinterpret_cast<const float2*>(x);
        float2* w = static_cast<float2*>(work);
        if (mis) {
            if (cudaMemcpyAsync(w, x, sizeof(float) * n, cudaMemcpyDeviceToDevice, st) != cudaSuccess) rc = -1;
            z = w;
            w += K + (K & 1);
        }
        if (!rc) rc = r2c_with(owner, *l, z, K, out, w, st);
    }
    // a length or working array too large to keep
    if (keep && l && l->bytes > kLengthBytes) drop_length(e, e.lengths.find(K), st);
    if (keep && e.work_bytes > kLengthBytes) drop_work(e, st);
    if (!keep) {
        once.release(st);
        e.plans.swap(once.plans);
    }
    return rc;
}

}  // namespace accel
