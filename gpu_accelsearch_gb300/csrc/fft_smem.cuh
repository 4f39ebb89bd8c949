// fft_smem.cuh -- complex FP32 FFT of M = 2^k points (64 <= M <= 8192) in
// shared memory, radix-16 passes plus one radix-2/4/8 pass.  T = M/16 threads
// each hold 16 points in registers; register e of thread t is point t + e*T
// both on entry (time order) and on exit (frequency order), so loads from and
// stores to global memory coalesce.
//
// Between passes the points go through shared memory, in place: a pass reads
// and writes the same 16 (or Q x R) positions, so only its writes need a
// barrier before the next pass reads them, one barrier per exchange.  With
// n = n1 + ... over the passes' digits, the first pass (over the top digit)
// leaves digit k1 of the frequency selecting a block of M/16 points, the
// second turns the next digit of n into k2 in place, and so on; the last
// pass's thread k = k1 + 16 k2 + ... then holds the points of frequency
// k + j M/R, R consecutive positions (16-byte reads).  The blocks are
// M/16 + 2 points apart (swizzled at 2048 points), and the threads of a middle
// pass take n1 and some bits of k1 along a half-warp, so that every access falls
// in 32 different banks.
// The butterflies and twiddles are those of the Stockham auto-sort form this
// replaces (the results are bit-identical), which needed a barrier between
// every pass's reads and writes as well and one after the last reads.  Plane
// kernels, us per segment of 656 rows (300 at 8192): 8192 points 13.95 -> 12.95,
// 4096 10.52 -> 10.38, 2048 4.46 -> 4.43, 512 0.66 -> 0.64.  (A barrier before
// the middle pass's butterflies, or the template pairs (A, B) side by side
// for 16-byte loads, help 4096 points by under 1 % and cost 2048 up to 3 %.)
//
// NB independent transforms of the same length are done side by side by
// the same threads (one barrier per pass for all of them), each through its
// own buffer: a transform's butterflies run while the other's shared-memory
// stores and loads are still in flight.
//
// Twiddles come from a table tw[m] = exp(+2 pi i m / kTwN) in global
// memory (computed once from double precision); the forward direction uses
// its conjugate.
#pragma once

#include "accel_common.cuh"

namespace accel {

__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 4); }

// Barrier between passes: the whole CTA (the default), or a named barrier
// over the group of threads doing one transform (several transforms of a
// smaller size side by side in one CTA, each group on its own barrier).
struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
struct GroupSync {
    int id, nthreads;  // barrier 1..15, a multiple of 32 threads
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(nthreads) : "memory");
    }
};
struct LaneSync {  // transforms of fewer than 32 threads: some lanes of one warp
    unsigned mask;
    __device__ __forceinline__ void operator()() const { __syncwarp(mask); }
};
template <int M> struct FftShape {
    static constexpr int T = M / 16;
    // 2048 points: blocks M/16 points apart, position i of block k1 kept at
    // i ^ 2 (k1 & 7), as free of bank conflicts as the padding.  The buffers of
    // four plane CTAs then fit the 132 KB shared-memory configuration (the
    // padded ones miss it by 2 KB) and the L1 has 124 KB instead of 92: plane
    // kernel with bulk row stores 4.30 -> 4.18 us per segment.  At the other
    // lengths the configuration stays the same either way.
    static constexpr bool SWZ = M == 2048;
    static constexpr int PITCH = SWZ ? M / 16 : M / 16 + 2;  // from one block of M/16 points to the next
    static constexpr int PADDED = 16 * PITCH;
};

// Sums and scaled sums of complex numbers, PK: both components in one packed
// instruction (add/sub/fma.rn.f32x2, the same roundings as two).  A packed
// instruction holds the FP32 pipe as long as two, so what it saves is issue
// slots: 54 -> 45 instructions per point, which moves the plane kernels 2 to 3
// % (their L1 data pipe is the busier unit).  The 8192-point transform keeps the
// scalar forms: both transforms of a row in one CTA, 16 warps and nothing else
// on the SM, measured 3 % slower packed (that form serves options only now; the
// default k_plane_half took the scalar sums over and was not measured packed).
template <bool PK> __device__ __forceinline__ float2 padd(float2 a, float2 b) {
    if constexpr (!PK) return cadd(a, b);
    float2 r;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 x, x, y;\n"
        " mov.b64 {%0, %1}, x;\n}\n"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
template <bool PK> __device__ __forceinline__ float2 psub(float2 a, float2 b) {
    if constexpr (!PK) return csub(a, b);
    float2 r;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 x, x, y;\n"
        " mov.b64 {%0, %1}, x;\n}\n"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
template <bool PK> __device__ __forceinline__ float2 pfma(float s, float2 a, float2 b) {  // s a + b
    if constexpr (!PK) return make_float2(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y));
    float2 r;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %2};\n mov.b64 y, {%3, %4};\n mov.b64 z, {%5, %6};\n"
        " fma.rn.f32x2 x, x, y, z;\n mov.b64 {%0, %1}, x;\n}\n"
        : "=f"(r.x), "=f"(r.y)
        : "f"(s), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// x * (DIR * i)
template <int DIR> __device__ __forceinline__ float2 mul_i(float2 a) {
    return DIR > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <int DIR> __device__ __forceinline__ void dft2(float2* v) {
    float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}

template <int DIR, bool PK> __device__ __forceinline__ void dft4(float2* v) {
    float2 s02 = padd<PK>(v[0], v[2]), d02 = psub<PK>(v[0], v[2]);
    float2 s13 = padd<PK>(v[1], v[3]), d13 = mul_i<DIR>(psub<PK>(v[1], v[3]));
    v[0] = padd<PK>(s02, s13);
    v[2] = psub<PK>(s02, s13);
    v[1] = cadd(d02, d13);
    v[3] = csub(d02, d13);
}

__device__ __forceinline__ float2 cfma(float s, float2 a, float2 b) {  // s a + b
    return make_float2(fmaf(s, a.x, b.x), fmaf(s, a.y, b.y));
}

// 8 points as 2 x 4; the twiddles W8^1 = s (1 + i'), W8^3 = s (-1 + i')
// (i' = DIR i, s = 1/sqrt2) applied by the fused multiply-adds of the last
// layer: 52 floating-point instructions instead of 56.
template <int DIR, bool PK> __device__ __forceinline__ void dft8(float2* v) {
    const float S = 0.70710678118654752440f;
    float2 e[4] = {v[0], v[2], v[4], v[6]};
    float2 o[4] = {v[1], v[3], v[5], v[7]};
    dft4<DIR, PK>(e);
    dft4<DIR, PK>(o);
    const float2 p1 = cadd(o[1], mul_i<DIR>(o[1])), p3 = csub(mul_i<DIR>(o[3]), o[3]);
    const float2 o2 = mul_i<DIR>(o[2]);
    v[0] = padd<PK>(e[0], o[0]), v[4] = psub<PK>(e[0], o[0]);
    v[1] = pfma<PK>(S, p1, e[1]), v[5] = pfma<PK>(-S, p1, e[1]);
    v[2] = cadd(e[2], o2), v[6] = csub(e[2], o2);
    v[3] = pfma<PK>(S, p3, e[3]), v[7] = pfma<PK>(-S, p3, e[3]);
}

// 16 points as 4 x 4: x[4 n1 + n2] -> X[k1 + 4 k2].  DFT4 over n1 for each
// n2, twiddles W16^(n2 k1), DFT4 over n2 for each k1.  Each nontrivial
// twiddle is written as a real scale times a factor with a unit component
// -- W^2 = s (1 + i'), W^6 = s (-1 + i'), W^1 = c (1 + t i'), W^3 =
// c (t + i'), W^9 = -c (1 + t i') with i' = DIR i, s = 1/sqrt2,
// c = cos(pi/8), t = tan(pi/8) -- and the scale is applied by the fused
// multiply-adds of the second DFT4 layer, whose two inputs of a pair carry
// the same scale: 144 floating-point instructions per 16 points instead of
// 160 with the twiddles multiplied out.
template <int DIR, bool PK> __device__ __forceinline__ void dft16(float2* v) {
    const float C = 0.92387953251128675613f, S = 0.70710678118654752440f, TN = 0.41421356237309504880f;
    float2 y[4][4];  // y[n2][k1]
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) {
        float2 u[4] = {v[n2], v[n2 + 4], v[n2 + 8], v[n2 + 12]};
        dft4<DIR, PK>(u);
#pragma unroll
        for (int k1 = 0; k1 < 4; k1++) y[n2][k1] = u[k1];
    }
    {  // k1 = 0: no twiddles
        float2 u[4] = {y[0][0], y[1][0], y[2][0], y[3][0]};
        dft4<DIR, PK>(u);
        v[0] = u[0], v[4] = u[1], v[8] = u[2], v[12] = u[3];
    }
    {  // k1 = 1: W^1 = c (1 + t i'), W^2 = s (1 + i'), W^3 = c (t + i')
        const float2 p2 = cadd(y[2][1], mul_i<DIR>(y[2][1]));
        const float2 s02 = pfma<PK>(S, p2, y[0][1]), d02 = pfma<PK>(-S, p2, y[0][1]);
        const float2 i1 = mul_i<DIR>(y[1][1]), i3 = mul_i<DIR>(y[3][1]);
        const float2 a1 = cfma(TN, i1, y[1][1]), a3 = cfma(TN, y[3][1], i3);
        const float2 s13 = padd<PK>(a1, a3), d13 = mul_i<DIR>(psub<PK>(a1, a3));
        v[1] = pfma<PK>(C, s13, s02), v[9] = pfma<PK>(-C, s13, s02);
        v[5] = cfma(C, d13, d02), v[13] = cfma(-C, d13, d02);
    }
    {  // k1 = 2: W^2 = s (1 + i'), W^4 = i', W^6 = s (-1 + i')
        const float2 i2 = mul_i<DIR>(y[2][2]);
        const float2 s02 = cadd(y[0][2], i2), d02 = csub(y[0][2], i2);
        const float2 a = psub<PK>(y[1][2], y[3][2]), ib = mul_i<DIR>(padd<PK>(y[1][2], y[3][2]));
        const float2 s13 = cadd(a, ib), d13 = csub(ib, a);
        v[2] = pfma<PK>(S, s13, s02), v[10] = pfma<PK>(-S, s13, s02);
        v[6] = pfma<PK>(S, d13, d02), v[14] = pfma<PK>(-S, d13, d02);
    }
    {  // k1 = 3: W^3 = c (t + i'), W^6 = s (-1 + i'), W^9 = -c (1 + t i')
        const float2 p2 = csub(mul_i<DIR>(y[2][3]), y[2][3]);
        const float2 s02 = pfma<PK>(S, p2, y[0][3]), d02 = pfma<PK>(-S, p2, y[0][3]);
        const float2 i1 = mul_i<DIR>(y[1][3]), i3 = mul_i<DIR>(y[3][3]);
        const float2 a1 = cfma(TN, y[1][3], i1), a3 = cfma(TN, i3, y[3][3]);
        const float2 s13 = psub<PK>(a1, a3), d13 = mul_i<DIR>(padd<PK>(a1, a3));
        v[3] = pfma<PK>(C, s13, s02), v[11] = pfma<PK>(-C, s13, s02);
        v[7] = cfma(C, d13, d02), v[15] = cfma(-C, d13, d02);
    }
}

template <int R, int DIR, bool PK = true> __device__ __forceinline__ void dft(float2* v) {
    if constexpr (R == 2) dft2<DIR>(v);
    else if constexpr (R == 4) dft4<DIR, PK>(v);
    else if constexpr (R == 8) dft8<DIR, PK>(v);
    else dft16<DIR, PK>(v);
}

template <int DIR> __device__ __forceinline__ float2 twid(const float2* __restrict__ tw, int idx) {
    float2 w = __ldg(tw + idx);
    return DIR > 0 ? w : make_float2(w.x, -w.y);
}

// The base twiddles W^k, W^2k, W^4k, W^8k (W = exp(DIR 2 pi i / NR)) of
// pass index k: from the two planes of NR's packed section (16-byte loads
// of consecutive memory) or, for NR = kTwN, from the table itself.
struct Tw16 {
    float2 w1, w2, w4, w8;
};
template <int DIR>
__device__ __forceinline__ Tw16 load_tw16(const float2* __restrict__ tw, int k, int NR) {
    Tw16 r;
    if (NR == kTwN) {
        r.w1 = twid<DIR>(tw, k);
        r.w2 = twid<DIR>(tw, (2 * k) & (kTwN - 1));
        r.w4 = twid<DIR>(tw, (4 * k) & (kTwN - 1));
        r.w8 = twid<DIR>(tw, (8 * k) & (kTwN - 1));
        return r;
    }
    const float4* p = reinterpret_cast<const float4*>(tw + kTwN + tw_pack_off(NR)) + k;
    const float4 a = __ldg(p), b = __ldg(p + tw_pack_entries(NR));
    const float sg = DIR > 0 ? 1.f : -1.f;
    r.w1 = make_float2(a.x, sg * a.y);
    r.w2 = make_float2(a.z, sg * a.w);
    r.w4 = make_float2(b.x, sg * b.y);
    r.w8 = make_float2(b.z, sg * b.w);
    return r;
}

// v[nb][r] *= W^{r k} with W = exp(DIR 2 pi i / NR), for every transform nb.
// Base powers from load_tw16; the rest are one product away.
template <int R, int DIR, int NB>
__device__ __forceinline__ void apply_twiddles(float2 (&v)[NB][R], const float2* __restrict__ tw, int k,
                                               int NR) {
    static_assert(R <= 8, "radix-16 passes use apply_tw16");
    const Tw16 b = load_tw16<DIR>(tw, k, NR);
    float2 w[R];
    w[1] = b.w1;
    if constexpr (R >= 4) {
        w[2] = b.w2;
        w[3] = cmul(w[2], w[1]);
        if constexpr (R >= 8) {
            w[4] = b.w4;
            w[5] = cmul(w[4], w[1]);
            w[6] = cmul(w[4], w[2]);
            w[7] = cmul(w[4], w[3]);
        }
    }
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
        for (int r = 1; r < R; r++) v[nb][r] = cmul(v[nb][r], w[r]);
}

// v[nb][r] *= W^{rk} for the radix-16 pass with NR = 256, every power from
// its own table entry (no products).
template <int DIR, int NB>
__device__ __forceinline__ void apply_tw16_full256(float2 (&v)[NB][16], const float2* __restrict__ tw, int k) {
    const float2* f = tw + kTwN + kTwFull256 + k;
#pragma unroll
    for (int r = 1; r < 16; r++) {
        const float2 w = twid<DIR>(f, (r - 1) * 16);
#pragma unroll
        for (int nb = 0; nb < NB; nb++) v[nb][r] = cmul(v[nb][r], w);
    }
}

template <int NB>
__device__ __forceinline__ void apply_tw16(float2 (&v)[NB][16], const Tw16& p) {
    float2 w[16];
    w[1] = p.w1;
    w[2] = p.w2;
    w[3] = cmul(p.w2, p.w1);
    w[4] = p.w4;
    w[5] = cmul(p.w4, p.w1);
    w[6] = cmul(p.w4, p.w2);
    w[7] = cmul(p.w4, w[3]);
    w[8] = p.w8;
    w[9] = cmul(p.w8, p.w1);
    w[10] = cmul(p.w8, p.w2);
    w[11] = cmul(p.w8, w[3]);
    w[12] = cmul(p.w8, p.w4);
    w[13] = cmul(w[12], p.w1);
    w[14] = cmul(w[12], p.w2);
    w[15] = cmul(w[12], w[3]);
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
        for (int r = 1; r < 16; r++) v[nb][r] = cmul(v[nb][r], w[r]);
}

// Radix-16 pass over the top digit: registers (time order) to shared memory.
template <int M, int DIR, int NB>
__device__ __forceinline__ void fft_first(float2 (&a)[NB][16], float2* sm, int t) {
    using S = FftShape<M>;
#pragma unroll
    for (int nb = 0; nb < NB; nb++) {
        dft<16, DIR, (M < 8192)>(a[nb]);
#pragma unroll
        for (int r = 0; r < 16; r++) sm[nb * S::PADDED + (S::SWZ ? t ^ (2 * (r & 7)) : t) + r * S::PITCH] = a[nb][r];
    }
}

// A radix-16 pass in place on the positions p0 + r STRIDE (r even) and
// p1 + r STRIDE (r odd), its twiddles applied by tw(a).
template <int M, int STRIDE, int DIR, int NB, class Twiddle>
__device__ __forceinline__ void fft_middle(float2 (&a)[NB][16], float2* sm, int p0, int p1, Twiddle tw) {
    using S = FftShape<M>;
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
        for (int r = 0; r < 16; r++) a[nb][r] = sm[nb * S::PADDED + (r & 1 ? p1 : p0) + r * STRIDE];
    tw(a);
#pragma unroll
    for (int nb = 0; nb < NB; nb++) {
        dft<16, DIR, (M < 8192)>(a[nb]);
#pragma unroll
        for (int r = 0; r < 16; r++) sm[nb * S::PADDED + (r & 1 ? p1 : p0) + r * STRIDE] = a[nb][r];
    }
}

// The last pass, radix R over consecutive positions p + (r ^ x), Q = 16/R
// butterflies per thread QSTEP positions apart.  k is the index of the first one, the q-th's
// is k + q T; out(e, y) takes the transforms' points t + e T as they are
// formed.
template <int M, int R, int QSTEP, int DIR, int NB, class Out>
__device__ __forceinline__ void fft_last(float2 (&a)[NB][16], const float2* sm, const float2* __restrict__ tw, int p, int x,
                                         int k, const Tw16* pre, Out out) {
    using S = FftShape<M>;
    constexpr int Q = 16 / R;
#pragma unroll
    for (int nb = 0; nb < NB; nb++)
#pragma unroll
        for (int q = 0; q < Q; q++)
#pragma unroll
            for (int r = 0; r < R; r += 2) {
                const float4 v = *reinterpret_cast<const float4*>(sm + nb * S::PADDED + p + q * QSTEP + (S::SWZ ? r ^ x : r));
                a[nb][q + r * Q] = make_float2(v.x, v.y);
                a[nb][q + (r + 1) * Q] = make_float2(v.z, v.w);
            }
#pragma unroll
    for (int q = 0; q < Q; q++) {
        float2 v[NB][R];
#pragma unroll
        for (int nb = 0; nb < NB; nb++)
#pragma unroll
            for (int r = 0; r < R; r++) v[nb][r] = a[nb][q + r * Q];
        // each twiddle is formed once and applied to every transform
        if constexpr (R == 16 && M == 256) apply_tw16_full256<DIR, NB>(v, tw, k);
        else if constexpr (R == 16) apply_tw16<NB>(v, *pre);
        else apply_twiddles<R, DIR, NB>(v, tw, k + q * S::T, M);
#pragma unroll
        for (int nb = 0; nb < NB; nb++) dft<R, DIR, (M < 8192)>(v[nb]);
#pragma unroll
        for (int r = 0; r < R; r++) {
            float2 y[NB];
#pragma unroll
            for (int nb = 0; nb < NB; nb++) y[nb] = v[nb][r];
            out(q + r * Q, y);
        }
    }
}

// Full transform: radix-16 passes, the leftover factor (2, 4 or 8) last.
// t is the thread's index within the group of M/16 threads doing the
// transform(s); sm must hold NB * FftShape<M>::PADDED float2, one buffer per
// transform.  The twiddles of a radix-16 pass of 4096 points are loaded up
// front (for one transform, which has 80 registers, where they are used).  out(e, y) takes the points t + e T of the transforms.  Other threads
// may still be reading shared memory when this returns.
template <int M, int DIR, int NB, class Sync, class Out>
__device__ __forceinline__ void fft_run_to(float2 (&a)[NB][16], float2* sm, const float2* __restrict__ tw, int t,
                                           Sync sync, Out out) {
    static_assert(M >= kMinM && M <= kMaxM && (M & (M - 1)) == 0, "M must be a power of two");
    constexpr int PITCH = FftShape<M>::PITCH, T = FftShape<M>::T;
    if constexpr (M <= 256) {
        // k1 = t + q T; consecutive points of its block
        fft_first<M, DIR, NB>(a, sm, t);
        sync();
        fft_last<M, M / 16, T * PITCH, DIR, NB>(a, sm, tw, t * PITCH, 0, t, nullptr, out);
    } else if constexpr (M <= 4096) {
        constexpr int B2 = M / 256;  // points of n1
        // second pass: n1 and the high bits of k1 along a half-warp
        constexpr int LB = B2 == 2 ? 1 : B2 == 4 ? 2 : B2 == 8 ? 4 : 8;  // lowest bit of k1 along a half-warp
        const int n1 = t & (B2 - 1), u = t >> 4;
        const int k1 = ((t / B2) & (16 / B2 - 1)) * LB + (u & (LB - 1)) + (u / LB) * 8;
        Tw16 p2;
        if constexpr (M == 4096 && NB > 1) p2 = load_tw16<DIR>(tw, t, 4096);
        fft_first<M, DIR, NB>(a, sm, t);
        sync();
        constexpr bool SWZ = FftShape<M>::SWZ;
        // (swizzled: bit 3 of a position is the low bit of r, which 2 (k1 & 4) flips)
        const int g = SWZ ? 2 * (k1 & 4) : 0, pm = k1 * PITCH + (SWZ ? n1 ^ (2 * (k1 & 3)) : n1);
        fft_middle<M, B2, DIR, NB>(a, sm, pm + g, pm - g,
                                   [&](float2 (&v)[NB][16]) { apply_tw16_full256<DIR, NB>(v, tw, k1); });
        sync();
        if constexpr (M == 4096 && NB == 1) p2 = load_tw16<DIR>(tw, t, 4096);
        // last: k = t + q T = k1 + 16 k2
        const int f = SWZ ? 2 * (t & 7) : 0;
        fft_last<M, B2, (T / 16) * B2, DIR, NB>(a, sm, tw, (t & 15) * PITCH + (((t >> 4) * B2) ^ (f & 8)), f & 6, t,
                                                &p2, out);
    } else {  // 8192 = 16 x 16 x 16 x 2
        const int n1 = t & 31, k1 = t >> 5;
        // third pass: m1 (1 bit), the high bits of k1 along a half-warp, k2 = t / 32
        const int m1 = t & 1, q1 = ((t >> 1) & 7) + ((t >> 4) & 1) * 8, q2 = t >> 5;
        const Tw16 p2 = load_tw16<DIR>(tw, q1 + 16 * q2, 4096);
        fft_first<M, DIR, NB>(a, sm, t);
        sync();
        fft_middle<M, 32, DIR, NB>(a, sm, k1 * PITCH + n1, k1 * PITCH + n1,
                                   [&](float2 (&v)[NB][16]) { apply_tw16_full256<DIR, NB>(v, tw, k1); });
        sync();
        fft_middle<M, 2, DIR, NB>(a, sm, q1 * PITCH + 32 * q2 + m1, q1 * PITCH + 32 * q2 + m1,
                                  [&](float2 (&v)[NB][16]) { apply_tw16<NB>(v, p2); });
        sync();
        // last: k = t + 512 q = k1 + 16 k2 + 256 k3
        fft_last<M, 2, 4, DIR, NB>(a, sm, tw, (t & 15) * PITCH + 32 * ((t >> 4) & 15) + 2 * (t >> 8), 0, t, nullptr,
                                    out);
    }
}

// The same with the outputs left in the registers.  TAIL: shared memory may
// be rewritten as soon as this returns.
template <int M, int DIR, int NB, class Sync = CtaSync, bool TAIL = false>
__device__ __forceinline__ void fft_run(float2 (&a)[NB][16], float2* sm, const float2* __restrict__ tw,
                                        int t, Sync sync = Sync()) {
    // the points that y replaces have been taken by then
    fft_run_to<M, DIR, NB, Sync>(a, sm, tw, t, sync, [&](int e, const float2 (&y)[NB]) {
#pragma unroll
        for (int nb = 0; nb < NB; nb++) a[nb][e] = y[nb];
    });
    if constexpr (TAIL) sync();
}

}  // namespace accel
