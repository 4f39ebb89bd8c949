// refine.cu -- candidate refinement (the reference's optimizeCandidates
// stub, bpd_candidates.cu:24-27), kernels of accel_optimize_candidates.
//
// The power the plane kernels compute at fundamental-plane position (r, z)
// is |sum_j X[j] conj(F(r - j - z/2; z))|^2 over the 2 hw(z) bins j in
// [ceil(r) - hw, ceil(r) + hw), where X is the whitened spectrum and F the
// response that generate_z_response samples (bpd_subharmonics.cu:146-226):
//     F(x; z) = integral over u in [0, 1] of exp(i pi (2 x u + z u^2)).
// Here it is evaluated at any (r, z), for every harmonic k r / H, k z / H
// (k = 1..H) of a candidate, and the summed power is maximised on three
// nested 5 x 5 grids (steps 1/4, 1/16, 1/64 in r and 1, 1/4, 1/16 in z
// around the best point so far).
//
// With the sum and the integral exchanged, and a phase common to all bins
// dropped, the amplitude about a centre bin jc is
//     integral over v in [-1/2, 1/2] of
//         exp(-i pi (2 (r - jc) v + z v^2)) S(v),
//     S(v) = sum_m X[jc + m] exp(2 pi i m (v + 1/2)):
// S depends on the window of bins only, so it is evaluated once per node of
// a Gauss-Legendre rule (panels of 64 nodes, at most 72 radians of phase
// per half panel: the rule's error is then below 1e-12 of the integral) and
// every grid point costs one product per node.  A grid point's window
// differs from the core window common to all points by a few bins at its
// ends, added per node as prefix sums.  All in double precision.
//
// Evaluating F by Fresnel integrals at every bin of every grid point took
// about 8 M double-precision operations per harmonic at z = 200, in one CTA
// of four warps per candidate: 8.7 ms for 64 candidates of 1 to 8
// harmonics (double precision runs at 1/64 of the single-precision rate).
// This form takes about 1 M, spread over a cluster of eight CTAs per
// candidate: 0.5 ms for the same candidates (a call 8.70 -> 0.74 ms on a
// GB300).  What bounds it is the double-precision pipe (44 % busy) and the
// imbalance of a candidate's few hundred nodes over 32 warps.
#include <cooperative_groups.h>

#include "accel_internal.h"

namespace accel {

namespace cg = cooperative_groups;

constexpr int kRefCluster = 8;    // CTAs per candidate
constexpr int kRefThreads = 128;
constexpr int kRefGrid = 25;      // points of a level's 5 x 5 grid
constexpr int kRefEdge = 12;      // most bins a window extends past the core on one side
constexpr int kRefPitch = kRefThreads + 1;  // of the reduction buffer (double2)

// exp(i pi x)
__device__ __forceinline__ double2 cispi(double x) {
    double s, c;
    sincospi(x, &s, &c);
    return make_double2(c, s);
}
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 zconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

// Squared power normalisation of harmonic k of every candidate, as the
// search applies it to the candidate's step: the squared rsqrt of the
// segment's median power / ln 2 (bpd_search.cu:144-181).
constexpr int kNormThreads = 512;
constexpr int kNormKeys = kMaxM / kNormThreads;  // a segment has at most kMaxM bins
__global__ void __launch_bounds__(kNormThreads) k_refine_norms(const RefineArgs a) {
    __shared__ unsigned long long scratch[kSelectScratch];
    const OptCand& cand = a.in[blockIdx.x];
    const int k = blockIdx.y;
    if (k >= cand.numharm) return;
    const float2* __restrict__ X = a.spec[cand.trial];
    const long long nb = a.numbins[cand.trial];
    const int nd = cand.numdata[k];
    const long long lo = cand.lobin[k];
    uint32_t key[kNormKeys];
#pragma unroll
    for (int j = 0; j < kNormKeys; j++) {
        const int i = threadIdx.x + j * kNormThreads;
        const long long b = lo + i;
        const float2 v = i < nd && b >= 0 && b < nb ? X[b] : make_float2(0.f, 0.f);
        key[j] = i < nd ? __float_as_uint(power_exact(v)) : 0xffffffffu;
    }
    const uint32_t mk = block_select_reg<kNormThreads, kNormKeys>(key, nd, (nd - 1) / 2, scratch);
    if (threadIdx.x == 0) {
        const double nrm = (double)rsqrt_norm((float)((double)__uint_as_float(mk) / kLn2), a.exact_rsqrt);
        a.norm2[(size_t)blockIdx.x * kMaxHarm + k] = nrm * nrm;
    }
}

// Halfwidths over the f-dots z0 +- dz: z_halfwidth grows with |z|.
__device__ __forceinline__ void halfwidth_range(double z0, double dz, int* lo, int* hi) {
    const int a = z_halfwidth(z0 - dz), b = z_halfwidth(z0 + dz);
    *lo = (z0 - dz <= 0.0 && z0 + dz >= 0.0) ? z_halfwidth(0.0) : min(a, b);
    *hi = max(a, b);
}

// REFINE false: the powers at the candidates' own positions, one point without
// the grids' steps, window ends and node values (512 candidates of 8 harmonics
// at z = 100: 1.4 ms a call, 2.5 as a grid of 25 equal points).
template <bool REFINE>
__global__ void __launch_bounds__(kRefThreads) __cluster_dims__(kRefCluster, 1, 1)
    k_refine(const RefineArgs a, const RefineNodes nodes) {
    constexpr int G = REFINE ? kRefGrid : 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* red = reinterpret_cast<double2*>(smem_raw);  // [kRefGrid][kRefPitch]
    double2* edge = red + kRefGrid * kRefPitch;           // [2][kRefEdge + 1][kRefThreads]
    __shared__ double2 s_part[kMaxHarm * G];              // this CTA's share of every amplitude
    __shared__ double s_pow[kMaxHarm * G];
    __shared__ double s_tot[G];
    __shared__ double s_best[2];
    __shared__ int s_bg, s_move[2];
    cg::cluster_group cluster = cg::this_cluster();
    const int ci = blockIdx.x / kRefCluster, rank = (int)cluster.block_rank(), tid = threadIdx.x;
    const OptCand& cand = a.in[ci];
    const float2* __restrict__ X = a.spec[cand.trial];
    const long long nb = a.numbins[cand.trial];
    const int H = cand.numharm;
    // this CTA's share of the candidate's nodes (harmonic by harmonic)
    int ntot = 0;
    for (int k = 0; k < H; k++) ntot += cand.panels[k] * kRefineNodes;
    const int n_lo = (int)((long long)ntot * rank / kRefCluster);
    const int n_hi = (int)((long long)ntot * (rank + 1) / kRefCluster);
    double2* __restrict__ Sbuf = a.scratch + (size_t)cand.scratch_off * kRefineValues;
    if (tid == 0) {
        s_best[0] = cand.r;
        s_best[1] = cand.z;
    }
    __syncthreads();
    constexpr int levels = REFINE ? 3 : 1;
#pragma unroll 1
    for (int lv = 0; lv < levels; lv++) {
        const double dr = REFINE ? 0.25 / (double)(1 << (2 * lv)) : 0.0;
        const double dz = 4.0 * dr;
        const double r0 = s_best[0], z0 = s_best[1];
        for (int i = tid; i < kMaxHarm * G; i += kRefThreads) s_part[i] = make_double2(0.0, 0.0);
        __syncthreads();
        int base = 0;  // first node of harmonic k
#pragma unroll 1
        for (int k = 1; k <= H; k++) {
            const int P = cand.panels[k - 1], first = base, nk = P * kRefineNodes;
            base += nk;
            const int lo = max(n_lo, first), hi = min(n_hi, first + nk);
            if (lo >= hi) continue;  // uniform over the CTA
            // core window [cl, cr): bins every point of every level sums (the
            // grids reach 0.65625 in r and 2.625 in z)
            const double reach = REFINE ? 0.66 : 0.0, zreach = REFINE ? 2.63 * k / H : 0.0;
            const long long jc = (long long)rint(cand.r * k / H);
            int hmin, hmax;
            halfwidth_range(cand.z * k / H, zreach, &hmin, &hmax);
            const long long cl = (long long)ceil((cand.r + reach) * k / H) - hmin;
            const long long cr = (long long)ceil((cand.r - reach) * k / H) + hmin;
            // this level's centres: ceil(r) of the five columns takes the
            // values c0 and (they span at most one bin) c0 + 1
            const long long c0 = (long long)ceil((r0 - 2.0 * dr) * k / H);
            int ca[5], hb[5];  // column's centre - c0, row's halfwidth
#pragma unroll
            for (int g = 0; g < 5; g++) {
                ca[g] = (int)((long long)ceil((r0 + (g - 2) * dr) * k / H) - c0);
                hb[g] = z_halfwidth((z0 + (g - 2) * dz) * k / H);
            }
            const int hl = max(max(max(hb[0], hb[1]), max(hb[2], hb[3])), hb[4]);
            const int dl = (int)(cl - c0), dh = (int)(c0 - cr);
            const int nl = max(0, min(kRefEdge, dl + hl)), nr = max(0, min(kRefEdge, dh + ca[4] + hl));
            const double rl = r0 * k / H - (double)jc, zl = z0 * k / H;
            const double invp = 1.0 / P;
            double2 acc[G];
#pragma unroll
            for (int i = 0; i < G; i++) acc[i] = make_double2(0.0, 0.0);
            const int taps = (int)(cr - cl);
            const bool staged = taps <= kRefGrid * kRefPitch;
            if (lv == 0 && staged) {  // the core window in double (red is free here)
                for (int i = tid; i < taps; i += kRefThreads) {
                    const long long j = cl + i;
                    const float2 x = (j >= 0 && j < nb) ? __ldg(X + j) : make_float2(0.f, 0.f);
                    red[i] = make_double2((double)x.x, (double)x.y);
                }
                __syncthreads();
            }
#pragma unroll 1
            for (int n = lo + tid; n < hi; n += kRefThreads) {
                const int q = n - first, p = q / kRefineNodes, i = q % kRefineNodes;
                const double xg = i < kRefineNodes / 2 ? -nodes.x[i] : nodes.x[kRefineNodes - 1 - i];
                const double wg = nodes.w[i < kRefineNodes / 2 ? i : kRefineNodes - 1 - i];
                const double v = -0.5 + ((double)p + 0.5 * (1.0 + xg)) * invp, w = wg * 0.5 * invp;
                // a node's values between levels: S; exp(2 pi i (v + 1/2)) and
                // its powers at the window's ends; the phasors of the grid's
                // centre and of the finest steps in r and z
                double2* __restrict__ node = Sbuf + (size_t)n * kRefineValues;
                double2 S, e1, pl, pr, er0, ez0, sr, sz;
                if (lv == 0) {
                    e1 = cispi(2.0 * v + 1.0);
                    pl = cispi(2.0 * (double)(cl - jc) * (v + 0.5));
                    pr = cispi(2.0 * (double)(cr - jc) * (v + 0.5));
                    S = make_double2(0.0, 0.0);  // Horner from the top bin
                    for (int j = taps - 1; j >= 0; j--) {
                        double2 x;
                        if (staged) x = red[j];
                        else {
                            const long long g = cl + j;
                            const float2 xf = (g >= 0 && g < nb) ? __ldg(X + g) : make_float2(0.f, 0.f);
                            x = make_double2((double)xf.x, (double)xf.y);
                        }
                        S = make_double2(fma(S.x, e1.x, fma(-S.y, e1.y, x.x)), fma(S.x, e1.y, fma(S.y, e1.x, x.y)));
                    }
                    S = zmul(S, pl);
                    er0 = cispi(-2.0 * rl * v);
                    ez0 = cispi(-zl * (v * v));
                    if constexpr (!REFINE) {
                        const double2 f = make_double2(ez0.x * w, ez0.y * w), V = zmul(S, f);
                        acc[0].x = fma(V.x, er0.x, fma(-V.y, er0.y, acc[0].x));
                        acc[0].y = fma(V.x, er0.y, fma(V.y, er0.x, acc[0].y));
                        continue;
                    }
                    sr = cispi(-2.0 / 64 * k / H * v);
                    sz = cispi(-1.0 / 16 * k / H * (v * v));
                    node[0] = S, node[1] = e1, node[2] = pl, node[3] = pr;
                    node[6] = sr, node[7] = sz;
                } else {  // written by this thread
                    S = node[0], e1 = node[1], pl = node[2], pr = node[3];
                    er0 = node[4], ez0 = node[5], sr = node[6], sz = node[7];
                }
                // steps of this level, and (from level 1 on) the centre moved
                // to the last level's best point, steps of the last level
                double2 srl = sr, szl = sz;
#pragma unroll 1
                for (int m = lv; m < 2; m++) {
                    srl = zmul(srl, srl), srl = zmul(srl, srl);
                    szl = zmul(szl, szl), szl = zmul(szl, szl);
                }
                if (lv > 0) {
                    const double2 q2 = zmul(srl, srl), r4 = zmul(q2, q2), t2 = zmul(szl, szl), z4 = zmul(t2, t2);
                    for (int m = 0; m < abs(s_move[0]); m++) er0 = zmul(er0, s_move[0] > 0 ? r4 : zconj(r4));
                    for (int m = 0; m < abs(s_move[1]); m++) ez0 = zmul(ez0, s_move[1] > 0 ? z4 : zconj(z4));
                }
                node[4] = er0, node[5] = ez0;
                // prefix sums of the bins below cl and from cr on
                double2* el = edge + tid;
                double2* er = edge + (kRefEdge + 1) * kRefThreads + tid;
                double2 s = make_double2(0.0, 0.0);
                el[0] = s;
                for (int m = 1; m <= nl; m++) {
                    pl = zmul(pl, zconj(e1));
                    const long long j = cl - m;
                    if (j >= 0 && j < nb) {
                        const float2 x = __ldg(X + j);
                        s = zadd(s, zmul(make_double2((double)x.x, (double)x.y), pl));
                    }
                    el[m * kRefThreads] = s;
                }
                s = make_double2(0.0, 0.0);
                er[0] = s;
                for (int m = 1; m <= nr; m++) {
                    const long long j = cr + m - 1;
                    if (j >= 0 && j < nb) {
                        const float2 x = __ldg(X + j);
                        s = zadd(s, zmul(make_double2((double)x.x, (double)x.y), pr));
                    }
                    pr = zmul(pr, e1);
                    er[m * kRefThreads] = s;
                }
                // phasors of the grid's columns (r) and rows (z); weights in
                double2 ea[5], fb[5];
                ea[2] = er0;
                fb[2] = make_double2(ez0.x * w, ez0.y * w);
                ea[3] = zmul(ea[2], srl);
                ea[4] = zmul(ea[3], srl);
                ea[1] = zmul(ea[2], zconj(srl));
                ea[0] = zmul(ea[1], zconj(srl));
                fb[3] = zmul(fb[2], szl);
                fb[4] = zmul(fb[3], szl);
                fb[1] = zmul(fb[2], zconj(szl));
                fb[0] = zmul(fb[1], zconj(szl));
#pragma unroll 1
                for (int c = 0; c <= ca[4]; c++) {
                    double2 V[5];
#pragma unroll
                    for (int b = 0; b < 5; b++) {
                        const int il = max(0, min(nl, dl - c + hb[b])), ir = max(0, min(nr, dh + c + hb[b]));
                        V[b] = zmul(zadd(S, zadd(el[il * kRefThreads], er[ir * kRefThreads])), fb[b]);
                    }
#pragma unroll
                    for (int g = 0; g < 5; g++) {
                        if (ca[g] != c) continue;  // uniform
#pragma unroll
                        for (int b = 0; b < 5; b++) {
                            double2& t = acc[REFINE ? 5 * g + b : 0];
                            t.x = fma(V[b].x, ea[g].x, fma(-V[b].y, ea[g].y, t.x));
                            t.y = fma(V[b].x, ea[g].y, fma(V[b].y, ea[g].x, t.y));
                        }
                    }
                }
            }
            // sum over the threads that had a node
            const int act = min(kRefThreads, hi - lo);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < G; i++)
                if (tid < act) red[i * kRefPitch + tid] = acc[i];
            __syncthreads();
            if (tid < 4 * G) {
                const int i = tid >> 2, part = tid & 3;
                double2 t = make_double2(0.0, 0.0);
                for (int m = part; m < act; m += 4) t = zadd(t, red[i * kRefPitch + m]);
                // the four parts lie in one quad of lanes of a full or (last
                // warp) 4-lane group
                const unsigned quad = 0xfu << (tid & 28);
                t.x += __shfl_xor_sync(quad, t.x, 1);
                t.y += __shfl_xor_sync(quad, t.y, 1);
                t.x += __shfl_xor_sync(quad, t.x, 2);
                t.y += __shfl_xor_sync(quad, t.y, 2);
                if (part == 0) s_part[(k - 1) * G + i] = t;
            }
            __syncthreads();
        }
        cluster.sync();  // every CTA's share is complete
        for (int i = tid; i < H * G; i += kRefThreads) {
            double2 t = make_double2(0.0, 0.0);
            for (int c = 0; c < kRefCluster; c++) t = zadd(t, cluster.map_shared_rank(s_part, c)[i]);
            s_pow[i] = a.norm2[(size_t)ci * kMaxHarm + i / G] * (t.x * t.x + t.y * t.y);
        }
        cluster.sync();  // all shares read: they may be cleared again
        if (tid < G) {
            double p = 0.0;
            for (int k = 0; k < H; k++) p += s_pow[k * G + tid];
            s_tot[tid] = p;
        }
        __syncthreads();
        if (tid == 0) {
            int bg = G / 2;  // the centre unless something is strictly larger
            for (int g = 0; g < G; g++)
                if (s_tot[g] > s_tot[bg]) bg = g;
            s_bg = bg;
            if constexpr (REFINE) {
                s_move[0] = bg / 5 - 2;
                s_move[1] = bg % 5 - 2;
                s_best[0] = r0 + (bg / 5 - 2) * dr;
                s_best[1] = z0 + (bg % 5 - 2) * dz;
            }
        }
        __syncthreads();
    }
    if (rank == 0 && tid == 0) {
        OptOut o;
        o.r = s_best[0];
        o.z = s_best[1];
        for (int k = 0; k < kMaxHarm; k++) o.harm[k] = k < H ? (float)s_pow[k * G + s_bg] : 0.f;
        o.power = s_tot[s_bg];
        a.out[ci] = o;
    }
}

// Panels of the node rule for a harmonic at f-dot z: the phase over half a
// panel stays within 72 radians for every point of the three grids.
int refine_panels(double z, double zreach) {
    int hw = 0;
    for (double s : {-1.0, 1.0}) hw = std::max(hw, z_halfwidth(z + s * zreach));
    const double pi = 3.14159265358979323846;
    return (int)std::min(1e6, std::max(1.0, std::ceil((2 * pi * (hw + 3) + pi * (std::fabs(z) + zreach)) / 144.0)));
}

// Nodes and weights of the 64-point Gauss-Legendre rule on [-1, 1] (the
// positive nodes, largest first): Newton iteration on P_64.
const RefineNodes& refine_nodes() {
    static const RefineNodes n = [] {
        RefineNodes r{};
        const int N = kRefineNodes;
        for (int i = 0; i < N / 2; i++) {
            long double x = std::cos(3.14159265358979323846L * (i + 0.75L) / (N + 0.5L)), d = 1;
            for (int it = 0; it < 20; it++) {
                long double p0 = 1, p1 = x;
                for (int k = 2; k <= N; k++) {
                    const long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
                    p0 = p1;
                    p1 = p2;
                }
                d = N * (x * p1 - p0) / (x * x - 1);
                x -= p1 / d;
            }
            r.x[i] = (double)x;
            r.w[i] = (double)(2 / ((1 - x * x) * d * d));
        }
        return r;
    }();
    return n;
}

template <bool REFINE> static int refine_launch(const RefineArgs& a, cudaStream_t st) {
    constexpr size_t smem =
        sizeof(double2) * (kRefGrid * kRefPitch + (REFINE ? 2 * (kRefEdge + 1) * kRefThreads : 0));
    static std::atomic<unsigned long long> attr{0};
    int dev = 0;
    if (attr_pending(attr, &dev)) {
        if (cudaFuncSetAttribute(k_refine<REFINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess)
            return -1;
        attr_set(attr, dev);
    }
    k_refine<REFINE><<<a.n * kRefCluster, kRefThreads, smem, st>>>(a, refine_nodes());
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_refine(const RefineArgs& a, cudaStream_t st) {
    if (a.n <= 0) return 0;
    k_refine_norms<<<dim3(a.n, a.maxharm), kNormThreads, 0, st>>>(a);
    if (cudaGetLastError() != cudaSuccess) return -1;
    return a.refine ? refine_launch<true>(a, st) : refine_launch<false>(a, st);
}

}  // namespace accel
